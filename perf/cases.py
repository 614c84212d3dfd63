"""The work a user of the engine has it do, as cases whose passes can be timed.

Every case goes through a public entry point: the drop-in ``Gillespie.run`` (sampled and
every-event), the stateful run-time API, ensembles from host and from device memory, heterogeneous
batches, and the learned surrogate's training step and queries.  Networks, rate constants and run
lengths are those of the repository's benchmark, tests and examples, or random mass-action networks
of the same family over its range (8 to 200 species, 16 to 1000 reactions).
"""

import math

import numpy as np
import torch

import rebop_gb300 as rb
from rebop_gb300 import surrogate

# name -> (species, initial counts, reactions as (rate, reactants, products)); a text rate is an
# expression over species
NETS = {
    # epidemic: ~2e3 events a trajectory, ending in an absorbing state
    "sir": (["S", "I", "R"], {"S": 999, "I": 1},
            [(1e-4, ["S", "I"], ["I", "I"]), (0.01, ["I"], ["R"])]),
    # gene expression with dimerization: ~2e4 events a trajectory at t = 1
    "dimer": (["gene", "mRNA", "protein", "dimer"], {"gene": 1},
              [(25.0, ["gene"], ["gene", "mRNA"]), (1000.0, ["mRNA"], ["mRNA", "protein"]),
               (0.001, ["protein", "protein"], ["dimer"]), (0.1, ["mRNA"], []), (1.0, ["protein"], [])]),
    # circadian oscillator, 9 species and 16 reactions: ~3e3 events per unit of time
    "vilar": (["Da", "A", "Dpa", "Dr", "Dpr", "Ma", "Mr", "R", "C"], {"Da": 1, "Dr": 1},
              [(1.0, ["Da", "A"], ["Dpa"]), (1.0, ["Dr", "A"], ["Dpr"]), (50.0, ["Dpa"], ["Da", "A"]),
               (100.0, ["Dpr"], ["Dr", "A"]), (50.0, ["Da"], ["Da", "Ma"]), (0.01, ["Dr"], ["Dr", "Mr"]),
               (500.0, ["Dpa"], ["Dpa", "Ma"]), (50.0, ["Dpr"], ["Dpr", "Mr"]), (50.0, ["Ma"], ["Ma", "A"]),
               (5.0, ["Mr"], ["Mr", "R"]), (2.0, ["A", "R"], ["C"]), (1.0, ["C"], ["R"]), (10.0, ["Ma"], []),
               (0.5, ["Mr"], []), (1.0, ["A"], []), (0.2, ["R"], [])]),
    # enzyme kinetics with a saturating catalysis rate: mass action and a rate expression mixed
    "enzyme": (["E", "S", "ES", "P"], {"E": 50, "S": 500},
               [(0.01, ["E", "S"], ["ES"]), (0.1, ["ES"], ["E", "S"]),
                ("0.3 * ES * S / (40 + S)", ["ES"], ["E", "P"])]),
}
VILAR_EVENTS_PER_TIME = 2750.0
MM = [([1, 1, 0, 0], [-1, -1, 1, 0]), ([0, 0, 1, 0], [1, 1, -1, 0]), ([0, 0, 1, 0], [1, 0, -1, 1])]


def listed():
    return [
        # the first thing a user does: one sampled trajectory through the drop-in
        {"name": "run-sir", "kind": "run", "net": "sir", "tmax": 250.0, "steps": 250},
        # an interactive loop over the stateful run-time API
        {"name": "advance-sir", "kind": "advance", "net": "sir", "tmax": 100.0, "steps": 20},
        # every reaction of one trajectory (nb_steps = 0)
        {"name": "events-dimer", "kind": "events", "net": "dimer", "tmax": 0.4},
        # a small-network ensemble with many samples, results as ordinary arrays
        {"name": "ensemble-sir", "kind": "ensemble", "net": "sir", "n": 10_000, "tmax": 250.0, "steps": 250,
         "where": "host"},
        # the headline ensemble, results copied back into page-locked arrays
        {"name": "ensemble-dimer", "kind": "ensemble", "net": "dimer", "n": 100_000, "tmax": 1.0, "steps": 100,
         "where": "pinned"},
        # the oscillator at the size its benchmark runs it: few long trajectories
        {"name": "ensemble-vilar", "kind": "ensemble", "net": "vilar", "n": 100, "tmax": 200.0, "steps": 200,
         "where": "host"},
        # a network of middle size
        {"name": "ensemble-mid", "kind": "ensemble", "net": "random", "S": 12, "R": 24, "net_seed": 3, "n": 20_000,
         "tmax": 0.1, "steps": 50, "where": "device"},
        # a large network, results left on the device for further analysis
        {"name": "ensemble-large", "kind": "ensemble", "net": "random", "S": 200, "R": 1000, "net_seed": 20260104,
         "n": 3000, "tmax": 0.3, "steps": 20, "where": "device"},
        # rate expressions
        {"name": "ensemble-enzyme", "kind": "ensemble", "net": "enzyme", "n": 10_000, "tmax": 60.0, "steps": 30,
         "where": "host"},
        # parameter sets of one network and networks of uneven size in one launch
        {"name": "batch", "kind": "batch", "n_mm": 32, "traj_mm": 256, "n_rand": 24, "traj_rand": 192, "net_seed": 5,
         "steps": 100},
        # one optimiser step of the surrogate at its training batch size
        {"name": "surrogate-step", "kind": "train", "batch": 4096},
        # a parameter sweep answered by the surrogate: draws of the counts at every query
        {"name": "surrogate-draws", "kind": "sample", "queries": 16_384, "draws": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "advance", "events", "ensemble", "ensemble", "ensemble", "ensemble", "large", "large",
                       "batch", "train", "sample", "predict"])
    if kind == "run":
        net = rng.choice(["sir", "dimer", "enzyme"])
        top = {"sir": 250.0, "dimer": 0.5, "enzyme": 60.0}[net]
        return {"kind": "run", "net": net, "tmax": round(top * rng.uniform(0.2, 1.0), 3), "steps": _log_int(rng, 5, 400)}
    if kind == "advance":
        return {"kind": "advance", "net": "sir", "tmax": round(rng.uniform(20.0, 200.0), 2), "steps": rng.randint(3, 40)}
    if kind == "events":
        return {"kind": "events", "net": "dimer", "tmax": round(rng.uniform(0.1, 0.5), 3)}
    if kind == "ensemble":
        net = rng.choice(["sir", "dimer", "dimer", "vilar", "enzyme", "mid", "mid"])
        c = {"kind": "ensemble", "net": net, "where": rng.choice(["host", "pinned", "device"])}
        if net == "sir":
            c.update(n=_log_int(rng, 64, 40_000), tmax=round(rng.uniform(50, 250), 1), steps=_log_int(rng, 10, 250))
        elif net == "dimer":
            # a sweep gives every trajectory its own rate constants
            c.update(n=_log_int(rng, 256, 60_000), tmax=round(rng.uniform(0.2, 1.0), 3), steps=_log_int(rng, 1, 100),
                     sweep=rng.random() < 0.3)
        elif net == "vilar":
            c.update(n=_log_int(rng, 32, 4000), tmax=round(rng.uniform(5, 40), 1), steps=_log_int(rng, 10, 200))
        elif net == "enzyme":
            c.update(n=_log_int(rng, 64, 10_000), tmax=round(rng.uniform(10, 60), 1), steps=_log_int(rng, 5, 60))
        else:
            c.update(net="random", S=rng.randint(8, 16), R=rng.randint(17, 32), net_seed=rng.randint(1, 10**6),
                     n=_log_int(rng, 1000, 20_000), tmax=round(rng.uniform(0.02, 0.1), 3), steps=_log_int(rng, 5, 50))
        return c
    if kind == "large":
        S = _log_int(rng, 17, 200)
        return {"kind": "ensemble", "net": "random", "S": S, "R": S * rng.randint(2, 5), "net_seed": rng.randint(1, 10**6),
                "n": _log_int(rng, 300, 3000), "tmax": round(rng.uniform(0.05, 0.2) * 100 / S / 5, 5),
                "steps": _log_int(rng, 5, 50), "where": rng.choice(["host", "device"])}
    if kind == "batch":
        return {"kind": "batch", "n_mm": rng.randint(4, 36), "traj_mm": _log_int(rng, 16, 256),
                "n_rand": rng.randint(2, 24), "traj_rand": _log_int(rng, 16, 192), "net_seed": rng.randint(1, 10**6),
                "steps": _log_int(rng, 10, 100)}
    if kind == "train":
        return {"kind": "train", "batch": _log_int(rng, 200, 8192)}
    if kind == "sample":
        return {"kind": "sample", "queries": _log_int(rng, 1, 16_384), "draws": _log_int(rng, 10, 500)}
    return {"kind": "predict", "queries": _log_int(rng, 1, 65_536)}


# ------------------------------------------------------------------ networks
def _random_network(net_seed, S, R):
    """Mass-action network of order <= 2 that keeps its activity: mostly conversions and exchanges,
    a few inflows, degradations and bindings; rates log-uniform in [1e-4, 1e1], counts Poisson(200)."""
    rng = np.random.default_rng(net_seed)
    reactions = []
    for _ in range(R):
        order = int(rng.choice([0, 1, 2], p=[0.05, 0.5, 0.45]))
        if order == 0:
            n_prod = 1
        elif order == 1:
            n_prod = 1 if rng.random() < 0.9 else 0
        else:
            n_prod = 2 if rng.random() < 0.9 else 1
        exps, diff = [0] * S, [0] * S
        for sp in rng.integers(0, S, size=order):
            exps[int(sp)] += 1
            diff[int(sp)] -= 1
        for sp in rng.integers(0, S, size=n_prod):
            diff[int(sp)] += 1
        reactions.append((float(np.exp(rng.uniform(np.log(1e-4), np.log(1e1)))), exps, diff))
    return reactions, rng.poisson(200.0, size=S).astype(np.int64)


def _lowered(case):
    """(reactions as (rate, exponents, differences), initial counts) of the case's network."""
    if case["net"] == "random":
        return _random_network(case["net_seed"], case["S"], case["R"])
    names, init, reactions = NETS[case["net"]]
    low = []
    for k, reactants, products in reactions:
        e = [reactants.count(s) for s in names]
        low.append((k, e, [products.count(s) - x for s, x in zip(names, e)]))
    return low, np.array([init.get(s, 0) for s in names], dtype=np.int64)


def _network(case):
    low, x0 = _lowered(case)
    net = rb.Network(len(x0))
    for k, e, d in low:
        if isinstance(k, str):
            from rebop_gb300 import expr

            names = NETS[case["net"]][0]
            net.add_reaction(rb.Rate.expression(expr.parse(k).to_expr({s: i for i, s in enumerate(names)}, {})), d)
        else:
            net.add_reaction(rb.Rate.lma(k, e), d)
    return net, x0


def _dropin(case):
    s = rb.Gillespie()
    for k, reactants, products in NETS[case["net"]][2]:
        s.add_reaction(k, reactants, products)
    return s


def _seeds(seed, n):
    return np.random.default_rng([seed, 17]).integers(np.iinfo(np.uint64).max, size=n, dtype=np.uint64)


# ------------------------------------------------------------------ surrogate
def _queries(seed, n):
    """Query rows (log10 rate factors, t) over the surrogate's domain, t from its sample grid."""
    rng = np.random.default_rng([seed, 23])
    return np.concatenate([rng.uniform(-1, 1, (n, 5)), rng.integers(0, 101, (n, 1)) / 100.0], axis=1).astype(np.float32)


def _rate_equations(x):
    """(protein, dimer) of the dimer network's rate equations at queries x, Runge-Kutta in 64 bits."""
    x = np.asarray(x, dtype=np.float64)
    k = np.array(surrogate.RATES0) * 10.0 ** x[:, :5]
    h = x[:, 5] / surrogate.RRE_STEPS

    def rhs(y):
        m, p = y[:, 0], y[:, 1]
        a2, a3 = k[:, 1] * m, k[:, 2] * np.maximum(p, 0) * np.maximum(p - 1, 0)
        a5 = k[:, 4] * np.maximum(p, 0)
        return np.stack([k[:, 0] - k[:, 3] * m, a2 - 2 * a3 - a5, a3], axis=1)

    y = np.zeros((len(x), 3))
    for _ in range(surrogate.RRE_STEPS):
        k1 = rhs(y)
        k2 = rhs(y + 0.5 * h[:, None] * k1)
        k3 = rhs(y + 0.5 * h[:, None] * k2)
        k4 = rhs(y + h[:, None] * k3)
        y = np.maximum(y + h[:, None] / 6 * (k1 + 2 * k2 + 2 * k3 + k4), 0)
    return y[:, 1:]


def _tuples(seed, n):
    """Training tuples: features (u, t, b) and targets (counts, log residuals), counts Poisson around
    the rate equations as the simulated ones are."""
    rng = np.random.default_rng([seed, 29])
    x = _queries(seed, n)
    mean = _rate_equations(x)
    b = np.log1p(mean)
    counts = rng.poisson(np.minimum(mean, 1e6)).astype(np.float64)
    res = np.log(counts + rng.uniform(1e-3, 1.0, counts.shape)) - b
    return (np.concatenate([x, b], axis=1).astype(np.float32), np.concatenate([counts, res], axis=1).astype(np.float32))


def _model(seed):
    """A surrogate in the middle of its training: input scaling set, weights with a few steps' spread,
    the optimiser's moments filled."""
    model = surrogate.MDN(seed=seed % 1000)
    g = torch.Generator().manual_seed(seed)
    model.step = 500
    model.x_mean = torch.tensor([0, 0, 0, 0, 0, 0.5, 4.5, 3.0], dtype=torch.float32, device="cuda")
    model.x_std = torch.tensor([0.58] * 5 + [0.29, 2.0, 2.5], dtype=torch.float32, device="cuda")
    for b in model.b:
        b.copy_(0.05 * torch.randn(b.shape, generator=g))
    for w, m, v in list(zip(model.W, model.mW, model.vW)) + list(zip(model.b, model.mb, model.vb)):
        m.copy_(1e-3 * torch.randn(w.shape, generator=g))
        v.copy_(1e-5 * (0.5 + torch.rand(w.shape, generator=g)))
    return model


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "seed": seed}
    if kind in ("run", "events"):
        s["system"] = _dropin(case)
        s["init"] = NETS[case["net"]][1]
        if kind == "events":
            # the program's own record arrays: a trajectory fills as many rows as it has events
            s["time"] = np.zeros(65_536)
            s["counts"] = {n: np.zeros(65_536, dtype=np.int64) for n in NETS[case["net"]][0]}
    elif kind == "advance":
        low, x0 = _lowered(case)
        s["x0"] = x0
        s["g"] = rb.api.Gillespie.new_with_seed(x0, False, seed)
        for k, e, d in low:
            s["g"].add_reaction(rb.Rate.lma(k, e), d)
        s["times"] = [case["tmax"] * i / case["steps"] for i in range(1, case["steps"] + 1)]
    elif kind == "ensemble":
        s["net"], s["x0"] = _network(case)
        n, S = case["n"], len(s["x0"])
        s["seeds"] = _seeds(seed, n)
        shape = (case["steps"] + 1, S, n)
        if case.get("sweep"):
            k = np.array([r[0] for r in _lowered(case)[0]])
            s["rates"] = k * 10.0 ** np.random.default_rng([seed, 31]).uniform(-0.5, 0.5, (n, len(k)))
        if case["where"] == "pinned":
            s["out"] = torch.empty(shape, dtype=torch.int64, pin_memory=True).numpy()
        elif case["where"] == "device":
            s["d_x0"] = torch.from_numpy(s["x0"]).cuda()
            s["d_seeds"] = torch.from_numpy(s["seeds"].view(np.int64)).cuda()
            s["d_out"] = torch.empty(shape, dtype=torch.int64, device="cuda")
            s["d_events"] = torch.empty(n, dtype=torch.int64, device="cuda")
            if "rates" in s:
                s["d_rates"] = torch.from_numpy(s["rates"]).cuda()
    elif kind == "batch":
        b = rb.Batch()
        nets = [rb.Network(4)]
        for e, d in MM:
            nets[0].add_reaction(rb.Rate.lma(1.0, e), d)
        rng = np.random.default_rng(case["net_seed"])
        item_seeds = _seeds(seed, case["n_mm"] * case["traj_mm"] + case["n_rand"] * case["traj_rand"])
        at = 0
        for _ in range(case["n_mm"]):
            rates = np.exp(rng.uniform(np.log(1e-3), np.log(1e1), 3))
            x0 = [int(rng.integers(10, 101)), int(rng.integers(100, 1001)), 0, 0]
            b.add(nets[0], x0, item_seeds[at:at + case["traj_mm"]], 1.0, case["steps"], rates=rates)
            at += case["traj_mm"]
        for k in range(case["n_rand"]):
            S, R = int(rng.integers(8, 65)), int(rng.integers(16, 257))
            reactions, _ = _random_network(case["net_seed"] * 7919 + k, S, R)
            net = rb.Network(S)
            for r in reactions:
                net.add_reaction(rb.Rate.lma(r[0], r[1]), r[2])
            nets.append(net)
            b.add(net, rng.integers(0, 501, size=S), item_seeds[at:at + case["traj_rand"]], 1e-3, case["steps"])
            at += case["traj_rand"]
        s.update(batch=b, nets=nets, items=case["n_mm"] + case["n_rand"])
    elif kind == "train":
        s["model"] = _model(seed)
        x, y = _tuples(seed, case["batch"])
        s["x"], s["y"] = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    else:
        s["model"] = _model(seed)
        s["q"] = torch.from_numpy(_queries(seed, case["queries"])).cuda()
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind in ("run", "events"):
        ds = s["system"].run(s["init"], tmax=case["tmax"], nb_steps=case.get("steps", 0), rng=s["seed"])
        if kind == "run":
            return {"time": np.asarray(ds.time), "counts": {n: np.asarray(ds[n]) for n in NETS[case["net"]][0]}}
        n = min(len(ds.time), len(s["time"]))
        s["time"][:n] = ds.time[:n]
        for name, v in s["counts"].items():
            v[:n] = ds[name][:n]
        return {"n": n, "time": s["time"], "counts": s["counts"]}
    if kind == "advance":
        g = s["g"]
        g.seed(s["seed"])
        g.set_species(s["x0"])
        g.set_time(0.0)
        counts = []
        for t in s["times"]:
            g.advance_until(t)
            counts.append([g.get_species(k) for k in range(len(s["x0"]))])
        return {"time": g.get_time(), "counts": np.array(counts)}
    if kind == "ensemble":
        if case["where"] == "device":
            r = s.get("d_rates")
            s["net"].run_ensemble_device(case["n"], s["d_x0"].data_ptr(), False, s["d_seeds"].data_ptr(), case["tmax"],
                                         case["steps"], s["d_out"].data_ptr(),
                                         rates_ptr=0 if r is None else r.data_ptr(), rates_per_traj=r is not None,
                                         events_ptr=s["d_events"].data_ptr(),
                                         stream=torch.cuda.current_stream().cuda_stream)
            return {"counts": s["d_out"], "events": s["d_events"]}
        res = s["net"].run_ensemble(s["x0"], s["seeds"], case["tmax"], case["steps"], rates=s.get("rates"),
                                    out=s.get("out"))
        return {"time": res.times, "counts": res.counts, "events": res.events.view(np.int64)}
    if kind == "batch":
        st = s["batch"].run()
        return {"events": int(st["events"]), "counts": [s["batch"].counts(k) for k in range(s["items"])]}
    if kind == "train":
        m = s["model"]
        loss = m.train_step(s["x"], s["y"], 1e-3)
        return {"loss": loss, "W": m.W, "b": m.b, "mW": m.mW, "mb": m.mb, "vW": m.vW, "vb": m.vb, "Wb": m.Wb}
    if kind == "sample":
        return s["model"].sample_counts(s["q"], case["draws"], seed=s["seed"])
    return s["model"].predict_params(s["q"])


# ------------------------------------------------------------------ work
def _events(case):
    """Reaction events of one trajectory, from the rate equations (they set the mean)."""
    if case["net"] == "vilar":
        return VILAR_EVENTS_PER_TIME * case["tmax"]
    low, x0 = _lowered(case)
    if case["net"] == "enzyme":
        low[2] = (0.3, [0, 0, 1, 0], low[2][2])
    k = np.array([r[0] for r in low])
    e = np.array([r[1] for r in low])
    d = np.array([r[2] for r in low], dtype=np.float64)
    slots = [[s for s in range(e.shape[1]) for _ in range(row[s])] for row in e]
    a = np.array([(row + [-1, -1])[0] for row in slots])
    b = np.array([(row + [-1, -1])[1] for row in slots])
    x = np.append(x0.astype(np.float64), 1.0)
    n = 2000
    total, h = 0.0, case["tmax"] / n
    for _ in range(n):
        p = k * x[a] * x[b]
        total += p.sum() * h
        x[:-1] = np.maximum(x[:-1] + h * (p @ d), 0)
    return total


def work(case):
    kind = case["kind"]
    if kind == "batch":
        out = 8.0 * (case["steps"] + 1) * (case["n_mm"] * case["traj_mm"] * 4 + case["n_rand"] * case["traj_rand"] * 36)
        return {"bytes": out, "flops": case["n_mm"] * case["traj_mm"] * 200.0 * 14
                + case["n_rand"] * case["traj_rand"] * 1700.0 * 450}
    if kind in ("train", "sample", "predict"):
        mlp = 2.0 * (8 * 256 + 3 * 256 * 256 + 256 * 112)
        weights = mlp / 2
        if kind == "train":
            return {"bytes": case["batch"] * 48.0 + weights * (4 * 6 + 2), "flops": 3 * mlp * case["batch"]}
        q = case["queries"]
        rre = 4.0 * surrogate.RRE_STEPS * 60
        if kind == "predict":
            return {"bytes": q * (24.0 + 448) + 2 * weights, "flops": q * (mlp + rre)}
        return {"bytes": q * (24.0 + 8 * case["draws"]) + 2 * weights, "flops": q * (mlp + rre + 60.0 * case["draws"])}
    low, x0 = _lowered(case)
    n = case.get("n", 1)
    per_event = sum(sum(r[1]) for r in low) + 2 * len(low) + 4
    events = _events(case)
    rows = events if kind == "events" else case["steps"] + 1
    return {"bytes": n * (8.0 * rows * len(x0) + 16), "flops": n * events * per_event}


# ------------------------------------------------------------------ exact values
def _grid(case):
    return np.array([case["tmax"] * i / case["steps"] for i in range(case["steps"] + 1)])


def _head_loss(o, y):
    """Mean negative log-likelihood of the count-aware head, 64-bit torch."""
    nc, kt = surrogate.NC, surrogate.KT
    total = 0.0
    for sp in range(2):
        blk = o[:, sp * (nc + 3 * kt):(sp + 1) * (nc + 3 * kt)]
        n, res = y[:, sp], y[:, 2 + sp]
        c = torch.clamp(n, max=nc - 1).long()
        logp = torch.log_softmax(blk[:, :nc], 1).gather(1, c[:, None])[:, 0]
        w, mu = torch.log_softmax(blk[:, nc:nc + kt], 1), blk[:, nc + kt:nc + 2 * kt]
        sg = torch.nn.functional.softplus(blk[:, nc + 2 * kt:]) + 1e-3
        e = (res[:, None] - mu) / sg
        tail = torch.logsumexp(w - 0.5 * e * e - torch.log(sg) - 0.5 * math.log(2 * math.pi), 1)
        total = total - logp - torch.where(c == nc - 1, tail, torch.zeros_like(tail))
    return total.mean()


def exact(case, seed):
    kind = case["kind"]
    if kind == "run" or (kind == "ensemble" and case["where"] != "device"):
        return {"time": _grid(case)}
    if kind == "advance":
        return {"time": float(case["tmax"])}
    if kind == "predict":
        m = _model(seed)
        x = _queries(seed, case["queries"])
        h = torch.from_numpy(np.concatenate([x.astype(np.float64), np.log1p(_rate_equations(x))], axis=1)).cuda()
        h = (h - m.x_mean.double()) / m.x_std.double()
        for i, (w, b) in enumerate(zip(m.W, m.b)):
            h = h @ w.double().T + b.double()
            h = torch.nn.functional.silu(h) if i < len(m.W) - 1 else h
        return h
    if kind == "train":
        m = _model(seed)
        x, y = _tuples(seed, case["batch"])
        W = [w.double().requires_grad_() for w in m.W]
        b = [v.double().requires_grad_() for v in m.b]
        h = (torch.from_numpy(x).cuda().double() - m.x_mean.double()) / m.x_std.double()
        for i in range(len(W)):
            h = h @ W[i].T + b[i]
            h = torch.nn.functional.silu(h) if i < len(W) - 1 else h
        loss = _head_loss(h, torch.from_numpy(y).cuda().double())
        grads = torch.autograd.grad(loss, W + b)
        step = m.step + 1
        out = {"loss": loss.detach(), "W": [], "b": [], "mW": [], "mb": [], "vW": [], "vb": [], "Wb": []}
        moments = list(zip(m.mW, m.vW)) + list(zip(m.mb, m.vb))
        for i, (p, g, (m1, m2)) in enumerate(zip(W + b, grads, moments)):
            m1 = 0.9 * m1.double() + 0.1 * g
            m2 = 0.999 * m2.double() + 0.001 * g * g
            p = p.detach() - 1e-3 * (m1 / (1 - 0.9 ** step)) / (torch.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
            k = "W" if i < len(W) else "b"
            out[k].append(p)
            out["m" + k].append(m1)
            out["v" + k].append(m2)
            if k == "W":
                out["Wb"].append(p)
        return out
    return None
