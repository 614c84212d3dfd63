// Warp-per-trajectory SSA kernel for large networks (hundreds of species,
// thousands of reactions), where one trajectory's propensity pass is itself
// data-parallel work.
//
// Each step of rebop's direct method (gillespie.rs:315-344) recomputes every
// propensity and folds them left to right into cumulative sums
// (make_cumrates, gillespie.rs:357-364).  Here the 32 lanes of a warp own
// contiguous chunks of the reaction list and keep every propensity as a 64-bit
// fixed-point number (units of 2^-E, E chosen per trajectory so that the total
// fills 52 to 60 bits).  Integer sums are exact and associative, so
//   * after a reaction fires each lane re-evaluates only those of its own
//     reactions that read a changed species (a bit mask per reaction and
//     lane, SsaArgs::dep_tab) and adds the differences to its chunk sum: no
//     re-summation, no drift, nothing handed between lanes;
//   * one shuffle scan of the chunk sums (two adds a step) gives every
//     chunk's prefix and the total, a second one over the chunk that holds
//     total * U the chosen reaction.
// The clock is a 64-bit fixed-point number too, counted from the interval's
// start in units of 2^-58 of the interval.  The random words are generated
// ahead, 32 at a time, one kept per lane: the lanes then turn all 32 into
// Exp1 candidates at once, and a step picks up the two words it consumes with
// shuffles.  The clock arithmetic runs on every lane alike, so no decision has
// to be handed around.
//
// The reference's sums are a sequential binary64 fold, within (R + M + 2)
// 2^-53 of the exact sums; a fixed-point propensity is within (M + 1) 2^-44 of
// its own value plus 2 units of the exact one.  A decision whose operands lie
// farther apart than both bounds together is the reference's decision.  A
// close choice is redone for that step alone with the exact fold below;
// anything else -- a close clock comparison, a count outside [0, 2^23), a rate
// outside 2^-60 .. 2^60 -- re-runs the sample interval from its saved start
// with the exact step: lanes compute the binary64 propensities in the
// reference's multiply order and fold them in order lane after lane, lane 0
// draws in native binary64, so counts, event numbers and the random stream
// equal rebop's bit for bit.
//
// Bound: instruction issue and, at 16 warps per SM, the dependent chain of a
// step: 618 warp instructions per event at 60 % issue on 200 species and 1000
// reactions (1 216 at 71 % with float-pair sums), 10 000 trajectories of 6.0e4
// events each in 569 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "ssa_spec_body.cuh"

namespace rbg {

namespace {

constexpr int kWarpMaxWarps = 16;
// batch launches: small per-warp regions, so registers set the warps per SM
constexpr int kWarpMaxWarpsBatch = 24;

struct WarpLayout {
    size_t block_bytes, warp_bytes;
};

// Lane l owns the C = ceil(R / 32) reactions l*C .. l*C + C - 1.  Arrays the
// lanes walk together are stored lane-major -- reaction l*C + i at position
// i*32 + l -- so one step of the walk touches 32 consecutive words.
__host__ __device__ inline int warp_chunk(int R) { return (R + 31) / 32; }

// Every reaction of order <= 2 over fewer than 32767 species: propensities
// come from two-slot shapes (shape_word) and the factor list is not needed.
__host__ __device__ inline bool warp_shape2(const SsaArgs &a) { return a.max_mults <= 2 && a.S < 32767; }

// Shared memory: block tables (Exp1 tables, float-pair rates when shared,
// shapes or factors, jumps), then per warp: the generator at the word buffer's
// start and at the interval's, counts, fixed-point propensities (and
// float-pair rates when per trajectory).  The counts at the interval start go
// to global memory (SsaArgs::warp_cnt0).
constexpr size_t kWarpState = 96;  // generator states: buffer start, before its last word, interval start
__host__ __device__ inline WarpLayout warp_layout(const SsaArgs &a) {
    WarpLayout l;
    const size_t RP = 32 * (size_t)warp_chunk(a.R);     // lane-major positions
    size_t b = 16 * 256 + 8 * 257 + 8 * 256 + 8 * 256;  // zxk, zf, zd, xdf
    if (!a.batch) {  // a batch's networks stay in global memory
        b += 8 * RP;                                        // shared float-pair rates (lane-major)
        if (!warp_shape2(a)) b += 4 * RP * a.P;             // factors (lane-major), when shapes do not cover
        b += 4 * RP;                                        // two-slot reaction shapes (lane-major)
        b += 4 * (size_t)a.R * a.Q;                         // jumps: species, delta (16 bit each)
    }
    l.block_bytes = (b + 15) & ~(size_t)15;
    size_t w = kWarpState + 8 * (size_t)a.S;            // generator states, counts
    w += 4 * ((size_t)a.S + 1);                         // counts as floats, plus the constant 1
    w += 8 * RP + 8;                                    // propensities (lane-major), alignment
    if (a.rate_stride) w += 8 * RP;                     // per-trajectory float-pair rates
    const size_t wt = 8 * 32 * (2 * (size_t)a.tbatch_S + 4);  // a thread unit's counts, their copy, generator
    if (a.batch && wt > w) w = wt;
    l.warp_bytes = (w + 15) & ~(size_t)15;
    return l;
}

// Physical slot of the propensity at lane-major position pos
// (reaction l*C + i at i*32 + l): the lane bits are XORed with the row, so a
// row read by the 32 lanes (the chunk sums) and a column read by the 32 lanes
// (the walk through one lane's chunk to the chosen reaction) both touch 32
// distinct banks.  Without it every lane of the walk hit the same bank.
__device__ __forceinline__ int pz(int pos) { return pos ^ ((pos >> 5) & 31); }

__device__ __forceinline__ int64_t shfl_i64(int64_t v, int src) {
    return (int64_t)__shfl_sync(0xffffffffu, (long long)v, src);
}

// Inclusive sum over the lanes of a warp, over the nearest 2 * last lanes
// (16: all 32): the shuffle's own range predicate guards the two adds.
template <int D>
__device__ __forceinline__ void scan_step(int64_t &v) {
    asm volatile(
        "{\n .reg .u32 lo, hi, rl, rh;\n .reg .pred p;\n mov.b64 {lo, hi}, %0;\n"
        " shfl.sync.up.b32 rl|p, lo, %1, 0, 0xffffffff;\n shfl.sync.up.b32 rh, hi, %1, 0, 0xffffffff;\n"
        " @p add.cc.u32 lo, lo, rl;\n @p addc.u32 hi, hi, rh;\n mov.b64 %0, {lo, hi};\n}\n"
        : "+l"(v)
        : "n"(D));
}
__device__ __forceinline__ int64_t scan_i64(int64_t v, int width) {
    scan_step<1>(v);
    if (width > 2) scan_step<2>(v);
    if (width > 4) scan_step<4>(v);
    if (width > 8) scan_step<8>(v);
    if (width > 16) scan_step<16>(v);
    return v;
}

// The warp kernel's fixed-point numbers have 22 fraction bits below the part a
// 32-bit conversion reaches: v = floor(a) 2^22 + the rest.  64-bit conversions
// from and to float run on the FP64 pipe here and kept it 67 % busy; the
// 32-bit ones do not.
constexpr int kFxLow = 22;
constexpr int kFxLim = 52;  // single values stay below 2^52: a below 2^30

// round((h + l) 2^22) within one unit (and 2^-47 of the value) for a float pair
// with 0 <= h < 2^31, |l| <= 2^-20 h; l22 = 2^22 l.
__device__ __forceinline__ int64_t fx_from_df(float h, float l22) {
    const int a = __float2int_rz(h);
    const int b = __float2int_rn(__fmaf_rn(__fsub_rn(h, (float)a), 0x1p22f, l22));
    return (int64_t)a * (1 << kFxLow) + b;
}

// Float pair of 0 <= v < 2^57 within 2^-45 (v >= 2^47).
__device__ __forceinline__ DF df_from_fx(int64_t v) {
    const int hi = (int)(v >> 27);
    const float fh = __int2float_rz(hi);
    const int rest = hi - __float2int_rz(fh);  // below 2^6
    const int lo = (rest << 25) + (int)((uint32_t)v >> 2 & 0x1FFFFFFu);
    return DF{__fmul_rn(fh, 0x1p27f), __fmul_rn((float)lo, 4.0f)};
}

// u 2^-53 for 0 < u < 2^53 as a float pair, within 2^-47 of u itself however
// small it is.
__device__ __forceinline__ DF df_u53_rel(uint64_t u) {
    const int z = __clzll((long long)u);
    const uint64_t v = u << z;
    const float s = __uint_as_float((uint32_t)(127 - 13 - z) << 23);
    return DF{__fmul_rn((float)(uint32_t)(v >> 40), s),
              __fmul_rn((float)((uint32_t)(v >> 16) & 0xFFFFFFu), __fmul_rn(s, 0x1p-24f))};
}

// 2^e for -126 <= e <= 126.
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }
// floor(log2(v)) of a positive normal float / double.
__device__ __forceinline__ int ilog2f(float v) { return (int)(__float_as_uint(v) >> 23) - 127; }
__device__ __forceinline__ int ilog2d(double v) { return (int)((uint64_t)__double_as_longlong(v) >> 52) - 1023; }

__device__ __forceinline__ double shfl_d(double v, int src) {
    return __longlong_as_double(__shfl_sync(0xffffffffu, __double_as_longlong(v), src));
}

// Exact binary64 propensity of reaction r in the reference's multiply order:
// Rate::rate's fold (gillespie.rs:71-90), or the macro's integer falling
// factorials (gillespie_macro.rs:133-146).
template <bool MACRO>
__device__ __forceinline__ double exact_propensity(const SsaArgs &it, const int64_t *cnt, double rate, int r) {
    double acc = rate;
    for (int p = 0; p < it.P; ++p) {
        const int o = it.fac_ord[r * it.P + p];
        if (o == 0) continue;
        const int64_t n = cnt[it.fac_sp[r * it.P + p]];
        if (MACRO) {
            int64_t ff = n;
            for (int j = 1; j < o; ++j) ff *= n - j;
            acc = __dmul_rn(acc, (double)ff);
        } else {
            for (int j = o - 1; j >= 0; --j) acc = __dmul_rn(acc, (double)(n - j));
        }
    }
    return acc;
}

// Exact binary64 propensities and their running sums, in scr: this warp's
// shared-memory scratch of 32 * ceil(R / 32) doubles, lane-major like the
// chunks.  Lane l evaluates and folds its own reactions l*C .. l*C + C - 1, in
// order, starting from the running sum lane l - 1 hands over, so the sums are
// the reference's sequential fold (make_cumrates, gillespie.rs:357-364) while
// every lane reads only its own column.  Returns the total on every lane.
template <bool MACRO>
__device__ __forceinline__ double warp_exact_fold(const SsaArgs &it, const int64_t *cnt, const double *rates,
                                                  double *scr) {
    const int lane = threadIdx.x & 31, R = it.R, C = warp_chunk(R);
    const int r_lo = min(R, lane * C), n_own = min(R, r_lo + C) - r_lo;
    for (int i = 0; i < n_own; ++i) scr[i * 32 + lane] = exact_propensity<MACRO>(it, cnt, rates[r_lo + i], r_lo + i);
    // one lane's chunk after the other; loads go ahead in blocks of 8
    double run = 0.0;
    for (int l = 0; l < 32; ++l) {
        if (lane == l) {
            for (int i0 = 0; i0 < n_own; i0 += 8) {
                double v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = i0 + j < n_own ? scr[(i0 + j) * 32 + lane] : 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (i0 + j < n_own) {
                        run = __dadd_rn(run, v[j]);
                        scr[(i0 + j) * 32 + lane] = run;
                    }
            }
        }
        run = shfl_d(run, l);
    }
    return run;
}

// The reaction the reference picks for `chosen` from the running sums in scr:
// #{r : cum_r < chosen} (gillespie.rs:402-407), or for define_system! the
// first r with chosen < cum_r (gillespie_macro.rs:150-171); R if none.
template <bool MACRO>
__device__ __forceinline__ int warp_exact_pick(const SsaArgs &it, const double *scr, double chosen) {
    const int lane = threadIdx.x & 31, R = it.R, C = warp_chunk(R);
    const int r_lo = min(R, lane * C), n_own = min(R, r_lo + C) - r_lo;
    if (MACRO) {
        int first = n_own;
        for (int i = n_own - 1; i >= 0; --i)
            if (chosen < scr[i * 32 + lane]) first = i;
        const unsigned int has = __ballot_sync(0xffffffffu, first < n_own);
        if (!has) return R;
        const int l = __ffs((int)has) - 1;
        return l * C + __shfl_sync(0xffffffffu, first, l);
    }
    int c = 0;
    for (int i = 0; i < n_own; ++i) c += scr[i * 32 + lane] < chosen ? 1 : 0;
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    return c;
}

// One exact step of the whole warp from the committed state (lane 0 holds the
// generator).  Returns 1 when a reaction fires (its index in idx, the clock in
// t), 0 when the step records the sample.
template <bool MACRO>
__device__ __noinline__ int warp_exact_step(const SsaArgs &it, const int64_t *cnt, const double *rates,
                                            const double *zig, double *scr, Xoshiro &g, double &t, double T,
                                            int &idx) {
    const int lane = threadIdx.x & 31;
    const double total = warp_exact_fold<MACRO>(it, cnt, rates, scr);
    int fire = 0;
    double chosen = 0.0;
    if (lane == 0 && 0.0 < total) {
        const double tn = __dadd_rn(t, __ddiv_rn(xo_exp1(g, zig, zig + kZigOffF), total));
        if (!(tn > T)) {
            fire = 1;
            t = tn;
            chosen = __dmul_rn(total, xo_uniform(g));
        }
    }
    fire = __shfl_sync(0xffffffffu, fire, 0);
    t = shfl_d(t, 0);
    if (!fire) return 0;
    idx = warp_exact_pick<MACRO>(it, scr, shfl_d(chosen, 0));
    return 1;
}

// The exact choice alone, for a step whose clock the float pairs decided
// (the reaction fires) but whose choice they left close: the reference's
// total, chosen = total * U for the uniform's top 53 bits u53, and the pick.
// Overwrites scr.
template <bool MACRO>
__device__ __noinline__ int warp_exact_choice(const SsaArgs &it, const int64_t *cnt, const double *rates,
                                              double *scr, uint64_t u53) {
    const double total = warp_exact_fold<MACRO>(it, cnt, rates, scr);
    const double chosen = __dmul_rn(total, __dmul_rn((double)u53, 0x1.0p-53));
    return warp_exact_pick<MACRO>(it, scr, chosen);
}

// Two-slot shape of reaction r (reactant order <= 2): slots (species, offset)
// 2A -> (A,0)(A,1); A+B -> (A,0)(B,0); A -> (A,0)(one); none -> (one)(one),
// species S standing for a constant 1.  The propensity is then
// rate * max(n1 - o1, 0) * max(n2 - o2, 0), without branches.
__host__ __device__ inline uint32_t shape_word(const int32_t *fac_sp, const int32_t *fac_ord, int P, int S, int r) {
    uint32_t sl[2] = {(uint32_t)S, (uint32_t)S}, of[2] = {0, 0};
    int k = 0;
    for (int p = 0; p < P; ++p) {
        const int o = fac_ord[r * P + p];
        for (int j = 0; j < o && k < 2; ++j, ++k) {
            sl[k] = (uint32_t)fac_sp[r * P + p];
            of[k] = (uint32_t)j;
        }
    }
    return sl[0] | of[0] << 15 | sl[1] << 16 | of[1] << 31;
}

// Exp1 draw as a float pair within gamma of itself, consuming the stream as
// the reference does (exp1_df with the candidate's fraction normalised first).
__device__ __forceinline__ DF exp1_df_rel(Xoshiro &g, const ExactTables &ex, const float2 *xdf) {
    for (;;) {
        const uint64_t b = xo_next(g);
        const int i = (int)(b & 0xff);
        const uint64_t k = b >> 12;
        const float2 X = xdf[i];
        const DF x = df_mul(df_u53_rel(2 * k + 1), DF{X.x, X.y});
        if (k < ex.zxk[i].y) return x;
        if (i == 0) return df_from_double(__dsub_rn(kZigR, log(xo_uniform(g))));
        if (wedge_df(ex, i, k, x.h, xo_next(g) >> 11)) return x;
    }
}

// One thread unit of a persistent batch: lane l runs trajectory first + l of
// the small-network item `it` (if it has one) from start to end with the
// speculative float-pair step of the thread kernels (ssa_spec_body.cuh):
// propensities as float pairs summed into a float32 running sum, the clock as
// a float triple with a rigorous error bound, the choice in float32 with an
// exact binary64 decision when it is close, and an exact re-run of any sample
// interval whose clock decision the bound leaves open -- so its counts,
// events and draws are rebop's.  wreg is this warp's region: counts [S][32],
// counts at the interval start [S][32] and the generator there [4][32].
// Returns the lane's event count; sets `late` if the wall-clock budget ran
// out (the trajectory is then incomplete).
// MAXR bounds the item's reactions (4, 8 or 16): the per-reaction loops are
// unrolled to it.
template <bool MACRO, int MAXR>
__device__ __noinline__ unsigned long long thread_unit(const SsaArgs &it, const ExactTables &zt, const float2 *xdf,
                                                       unsigned char *wreg, long long first, int64_t t_start,
                                                       bool &late) {
    using Ops = TableOps<MAXR, MACRO>;
    constexpr int NS = 32;  // column stride of the per-lane arrays
    const int lane = threadIdx.x & 31;
    const long long traj = first + lane;
    if (traj >= it.n_traj) return 0;
    const int S = it.S, R = it.R;
    int64_t *sp = reinterpret_cast<int64_t *>(wreg) + lane;
    int64_t *sps = sp + NS * S;
    uint64_t *gsv = reinterpret_cast<uint64_t *>(sps + NS * S);
    const ExactTables ex{zt.zxk, zt.zf, zt.zd, it.fac_packed, it.jmp_sp, it.jmp_d};
    for (int s = 0; s < S; ++s) sp[s * NS] = it.x0[traj * it.x0_stride + s];
    Xoshiro g;
    xo_seed(g, it.seeds[traj]);
    const uint64_t *rl = reinterpret_cast<const uint64_t *>(it.rate + traj * it.rate_stride);
    const float2 *rf = it.lm_rdf + traj * it.rate_stride;
    bool nat = false, exact_traj = false;
    for (int r = 0; r < R; ++r) {
        nat |= !emul_domain(rl[r]);
        exact_traj |= !spec_rate_ok(rl[r]);
    }
    exact_traj |= nat;
    // error model of the float-pair step (ssa_spec_body.cuh)
    const float G = ((float)(it.max_mults + R + 2) + (float)(R * (R + 1) / 2 + R * (it.max_mults + 2)) * 0.0625f) *
                    kGamma;
    const float c_q = G + 6.0f * kGamma;
    const float c_sel = (float)(it.max_mults + R + 6) * 0x1p-24f * 1.001f;
    typename Ops::Counts c{};
    unsigned long long ev = 0;
    uint64_t t0 = 0;  // clock at the interval start (bits)
    unsigned int tick = 0;
    for (long long i = 0; i < it.n_samples; ++i) {
        const double Td = it.sample_t[i];
        const uint64_t T = (uint64_t)__double_as_longlong(Td);
        const TF Tc = tf_from_double(Td);
        TF tc = tf_from_double(__longlong_as_double((long long)t0));
        float err_t = 0.0f;
        for (int s = 0; s < S; ++s) sps[s * NS] = sp[s * NS];
        gsv[0] = g.s0;
        gsv[NS] = g.s1;
        gsv[2 * NS] = g.s2;
        gsv[3 * NS] = g.s3;
        const unsigned long long ev0 = ev;
        bool replay = exact_traj;
        while (!replay) {
            if ((++tick & 1023u) == 0 && global_ns() - t_start > it.budget_ns) {
                late = true;
                return ev;
            }
            // both draws the step may make, taken ahead (stepped back when fewer
            // are committed)
            const uint64_t b1 = xo_next(g);
            const uint64_t b2 = xo_next(g);
            const int i1 = (int)(b1 & 0xff);
            const uint64_t k1 = b1 >> 12;
            const uint64_t K1 = ex.zxk[i1].y;
            const float2 X1 = xdf[i1];
            DF x = df_mul(df_u53(2 * k1 + 1), DF{X1.x, X1.y});
            float xerr = kGamma * X1.x;
            float cum[MAXR];
            DF tot;
            bool amb = Ops::props(it, ex, c, sp, NS, rf, 1, cum, tot);
            const bool slow = !(k1 < K1);
            uint64_t bu = b2;
            if (!(tot.h > 0.0f)) {
                xo_prev(g);  // no reaction can fire: no draw is made
                xo_prev(g);
                if (amb) replay = true;
                break;  // the sample records
            }
            if (slow) {
                x = exp1_df_cont(g, b1, b2, x, ex, xdf, xerr);
                bu = xo_next(g);
            }
            amb |= tot.h < 0x1p-90f || tot.h > 0x1p90f;
            const float rr = rcp_approx(tot.h);
            const DF q = df_div(x, tot, rr);
            const TF tn = tf_add(tc, q);
            float err_tn = __fadd_ru(err_t, __fmul_ru(c_q, q.h));
            err_tn = __fadd_ru(err_tn, __fmul_ru(__fmul_ru(xerr, rr), 1.001f));
            err_tn = __fadd_ru(err_tn, __fmul_ru(0x1p-52f, tn.h));
            err_tn = __fadd_ru(err_tn, __fmul_ru(0x1p-23f, fabsf(tn.l)));
            const float d = __fadd_rn(__fsub_rn(Tc.h, tn.h), __fadd_rn(__fsub_rn(Tc.m, tn.m), __fsub_rn(Tc.l, tn.l)));
            const float mt = __fadd_ru(err_tn, __fmul_ru(0x1p-44f, fmaxf(Tc.h, tn.h)));
            const float dd = __fmul_rn(d, 1.0f - 0x1p-22f);
            const bool fire = dd > mt;
            amb |= !(fire || dd < -mt) || !(err_tn < 1.0e30f) || q.h < 0x1p-100f;
            if (amb) {
                replay = true;
                break;
            }
            if (!fire) {
                xo_prev(g);  // the sample records: the Exp1 draw alone was made
                break;
            }
            const float ch = __fmul_rn(tot.h, f23((uint32_t)(bu >> 41)) * 0x1p-23f);
            const float msel = c_sel * tot.h;
            bool close = false;
            int idx = 0;
#pragma unroll
            for (int r = 0; r < MAXR; ++r) {
                if (r < R) {
                    const float dr = __fsub_rn(cum[r], ch);
                    idx += dr < 0.0f ? 1 : 0;
                    close |= fabsf(dr) <= msel;
                }
            }
            if (close) idx = Ops::exact_choice(it, ex, c, sp, NS, rl, 1, bu >> 11);
            tc = tn;
            err_t = err_tn;
            ++ev;
            Ops::jump(c, it, ex, sp, NS, idx);
        }
        if (replay) {
            // the interval again, exactly, from its saved start
            ev = replay_interval<MAXR, MACRO>(it, ex, sp, sps, gsv, rl, 1, NS, t0, T, nat, ev0, t_start);
            if (ev == ~0ull) {
                late = true;
                return ev0;
            }
            g = Xoshiro{gsv[0], gsv[NS], gsv[2 * NS], gsv[3 * NS]};
        }
        int64_t *o = it.out + (size_t)i * it.n_save * it.n_traj + traj;
        for (int k = 0; k < it.n_save; ++k) o[(size_t)k * it.n_traj] = sp[it.save_idx[k] * NS];
        t0 = T;  // the sample records at T (gillespie.rs:328-330)
    }
    if (it.events) it.events[traj] = ev;
    return ev;
}

// BATCH: the launch runs a.batch's networks (each item's tables in global
// memory, lane-major) and a.tbatch's thread units; otherwise the one network
// of `a`, whose tables the block copies to shared memory.
template <bool MACRO, bool BATCH>
__global__ void __launch_bounds__(32 * (BATCH ? kWarpMaxWarpsBatch : kWarpMaxWarps), 1)
    ssa_warp_kernel(const __grid_constant__ SsaArgs a) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const WarpLayout L = warp_layout(a);  // sized for the largest network of the launch

    // ---- block tables: Exp1 tables; in single-network mode also the
    // network's lane-major rates, factors, shapes and its jumps
    ulonglong2 *zxk = reinterpret_cast<ulonglong2 *>(g_spec_smem);
    uint64_t *zf = reinterpret_cast<uint64_t *>(zxk + 256);
    uint64_t *zd = zf + 257;
    float2 *xdf = reinterpret_cast<float2 *>(zd + 256);
    float2 *rdf_sh = xdf + 256;
    const int C0 = warp_chunk(a.R), RP0 = 32 * C0;
    const bool shape2 = warp_shape2(a);
    int32_t *facl_sh = reinterpret_cast<int32_t *>(rdf_sh + RP0);  // absent (size 0) when shape2
    uint32_t *shape_sh = reinterpret_cast<uint32_t *>(facl_sh + (shape2 ? 0 : (size_t)RP0 * a.P));
    // jumps of the one network: species as 16-bit indices (S < 65536) below
    // deltas of 16 bits when every one fits (else read from the descriptor)
    uint32_t *jump_sh = shape_sh + RP0;
    for (int k = tid; k < 256; k += blockDim.x) {
        zxk[k] = make_ulonglong2((uint64_t)__double_as_longlong(a.zig[k]),
                                 (uint64_t)__double_as_longlong(a.zig[kZigOffK + k]));
        zd[k] = (uint64_t)__double_as_longlong(a.zig[kZigOffD + k]) & ~(1ull << 63);
    }
    for (int k = tid; k < 257; k += blockDim.x) zf[k] = (uint64_t)__double_as_longlong(a.zig[kZigOffF + k]);
    bool jd_wide = false;
    if (!BATCH) {
        for (int k = tid; k < a.R * a.Q; k += blockDim.x) {
            const int64_t dlt = a.jmp_d[k];
            jump_sh[k] = (uint32_t)a.jmp_sp[k] | ((uint32_t)(uint16_t)dlt << 16);
            jd_wide |= dlt != (int64_t)(int16_t)dlt;
        }
        for (int q = tid; q < RP0; q += blockDim.x) {
            const int i = q >> 5, l = q & 31, r = l * C0 + i;
            if (!a.rate_stride) {
                const DF d = r < a.R ? df_from_double(a.rate[r]) : DF{0.f, 0.f};
                rdf_sh[q] = make_float2(d.h, d.l);
            }
            if (shape2) {
                shape_sh[q] = r < a.R ? shape_word(a.fac_sp, a.fac_ord, a.P, a.S, r) : (uint32_t)a.S << 16 | a.S;
            } else {
                for (int p = 0; p < a.P; ++p)
                    facl_sh[(i * a.P + p) * 32 + l] =
                        r < a.R ? (a.fac_sp[r * a.P + p] | (a.fac_ord[r * a.P + p] << 16)) : 0;
            }
        }
    }
    for (int k = tid; k < 256; k += blockDim.x) {
        const double v = a.zig[kZigOffXdf + k];
        xdf[k] = *reinterpret_cast<const float2 *>(&v);
    }
    jd_wide = __syncthreads_or(jd_wide);
    // the Exp1 draws use the ziggurat tables only
    const ExactTables ex{zxk, zf, zd, nullptr, nullptr, nullptr};

    // ---- this warp's region (sized for the largest network)
    unsigned char *wbase = g_spec_smem + L.block_bytes + (size_t)warp * L.warp_bytes;
    uint64_t *gst = reinterpret_cast<uint64_t *>(wbase);  // [12]: buffer start, before its last word, interval start
    int64_t *cnt = reinterpret_cast<int64_t *>(wbase + kWarpState);
    int64_t *cnt0 = a.warp_cnt0 + ((size_t)blockIdx.x * nw + warp) * (size_t)a.S;  // global
    float *cntf = reinterpret_cast<float *>(cnt + a.S);  // [S + 1]
    int64_t *prop = reinterpret_cast<int64_t *>((reinterpret_cast<uintptr_t>(cntf + a.S + 1) + 7) & ~(uintptr_t)7);
    float2 *rdf_w = reinterpret_cast<float2 *>(prop + RP0);  // per-trajectory float-pair rates (single-network mode)
    // exact steps use the propensity array as their scratch (32 * C doubles)
    double *scr = reinterpret_cast<double *>(prop);
    const int64_t t_start = global_ns();
    unsigned long long warp_events = 0;
    bool abort_run = false;

    for (;;) {
        long long ticket = 0;
        if (lane == 0) ticket = (long long)atomicAdd(a.work, 1ull);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket >= a.n_traj) break;

        // ---- a thread unit: 32 trajectories of a small network, one per lane
        if (BATCH && ticket >= a.n_warp_tickets) {
            const long long u = ticket - a.n_warp_tickets;
            int lo = 0, hi = a.tbatch_n - 1;  // last item with tbatch_unit <= u
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.tbatch_unit[mid] <= u) lo = mid;
                else hi = mid - 1;
            }
            bool late = false;
            const SsaArgs &ti = a.tbatch[lo];
            const long long first = (u - a.tbatch_unit[lo]) * 32;
            unsigned long long ev = ti.R <= 4   ? thread_unit<MACRO, 4>(ti, ex, xdf, wbase, first, t_start, late)
                                    : ti.R <= 8 ? thread_unit<MACRO, 8>(ti, ex, xdf, wbase, first, t_start, late)
                                                : thread_unit<MACRO, 16>(ti, ex, xdf, wbase, first, t_start, late);
            for (int off = 16; off > 0; off >>= 1) ev += __shfl_xor_sync(0xffffffffu, ev, off);
            warp_events += ev;
            if (__any_sync(0xffffffffu, late)) {
                if (lane == 0) atomicExch(a.work + 2, 1ull);
                break;
            }
            __syncwarp();
            continue;
        }

        // ---- the trajectory's network and run
        long long traj = ticket;
        const SsaArgs *itp = &a;
        if (BATCH) {
            int lo = 0, hi = a.batch_n - 1;  // last item with batch_start <= ticket
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.batch_start[mid] <= ticket) lo = mid;
                else hi = mid - 1;
            }
            itp = a.batch + lo;
            traj = ticket - a.batch_start[lo];
        }
        const SsaArgs &it = *itp;
        const int S = it.S, R = it.R, P = it.P, Q = it.Q;
        const int C = warp_chunk(R);
        const float2 *rdf = BATCH ? it.lm_rdf : (it.rate_stride ? rdf_w : rdf_sh);
        const int32_t *facl = BATCH ? it.lm_fac : facl_sh;
        const uint32_t *shape = BATCH ? it.lm_shape : shape_sh;
        const bool use_shape = BATCH ? it.lm_shape != nullptr : (it.max_mults <= 2 && it.S < 32767);
        // lane l owns reactions [l * C, min(R, (l + 1) * C)); local index i sits at i*32 + l
        const int r_lo = min(R, lane * C), r_hi = min(R, r_lo + C);
        const int n_own = r_hi - r_lo;
        const int mm = use_shape ? 2 : it.max_mults;  // multiplies per propensity
        // dependency masks; without them every propensity is re-evaluated
        const int dep_bytes = it.dep_bytes, n_words = (C + 31) >> 5;
        const void *dep_tab = it.dep_tab;
        // Fixed point: single propensities and the 32 chunk sums stay below
        // 2^52, so nothing overflows (up to 256 reactions a lane); the total is
        // scaled to 2^50 .. 2^51, and scaled anew when it falls below 2^47 or a
        // chunk sum reaches 2^52.
        // Relative error bound of a propensity or sum against the reference's
        // binary64 one, apart from one unit per propensity:
        const float c_p = (float)(mm + 2) * kGamma + (float)(R + mm + 4) * 0x1p-53f;
        // Exp1 / total: the total's bound (its units at the smallest total),
        // the Exp1 pair, the total's pair and the division
        const float c_q = (c_p + (float)(R + 2) * 0x1p-47f + 9.0f * kGamma) * 1.001f;
        const int sh_q = -ilog2f(c_q) - 1;         // 2^-sh_q >= c_q
        const int sh_p = -ilog2f(2.0f * c_p) - 1;  // choice: both operands' bounds
        // fixed-point propensity of the reaction at lane-major position pos, sc
        // times its value in units of 2^-22; mx collects the largest count it read (as float
        // bits: a count outside [0, 2^23) has bits >= 0x4B000000), mh the
        // largest sc * propensity
        auto eval_prop = [&](int pos, float sc, uint32_t &mx, float &mh) -> int64_t {
            const float2 k = rdf[pos];
            DF acc{k.x, k.y};
            if (use_shape) {
                const uint32_t w = shape[pos];  // the first slot's offset is 0
                const float n1 = cntf[w & 0x7FFFu], n2 = cntf[(w >> 16) & 0x7FFFu];
                mx = max(mx, max(__float_as_uint(n1), __float_as_uint(n2)));
                acc = df_mul_fu(df_mul_fu(acc, n1), fmaxf(__fsub_rn(n2, (float)(w >> 31)), 0.0f));
            } else {
                const int i2 = pos >> 5, l = pos & 31;
                for (int p = 0; p < P; ++p) {
                    const int f = facl[(i2 * P + p) * 32 + l];
                    const int o = f >> 16;
                    if (o == 0) continue;
                    const float n = cntf[f & 0xFFFF];
                    mx = max(mx, __float_as_uint(n));
                    for (int j = 0; j < o; ++j) acc = df_mul_fu(acc, fmaxf(__fsub_rn(n, (float)j), 0.0f));
                    acc = fast2sum(acc.h, acc.l);
                }
            }
            const float hs = __fmul_rn(acc.h, sc);
            mh = fmaxf(mh, hs);
            return fx_from_df(hs, __fmul_rn(acc.l, __fmul_rn(sc, 0x1p22f)));
        };
        bool need_full = true;  // every propensity to be evaluated, the scale chosen anew
        bool amb_next = false;  // a re-evaluated propensity read a count out of range
        bool absorbed = false;  // every propensity is 0
        float sc = 1.0f;        // scale of the fixed point
        int64_t ls = 0;         // this lane's chunk sum

        // ---- start (or resume) the trajectory.  g (the same on every lane) is
        // the generator past the word buffer, word p of which comes next
        // (p = 32: empty); x and acc_mask are the words' Exp1 candidates and
        // which of them the ziggurat's first test accepts.
        Xoshiro g;
        int p = 32;
        uint64_t word = 0;
        DF x{0.f, 0.f};
        uint32_t acc_mask = 0;
        double t;
        if (it.in_species) {
            for (int s = lane; s < S; s += 32) cnt[s] = it.in_species[traj * S + s];
            t = it.in_t[traj];
            g = Xoshiro{it.in_rng[traj * 4], it.in_rng[traj * 4 + 1], it.in_rng[traj * 4 + 2], it.in_rng[traj * 4 + 3]};
        } else {
            for (int s = lane; s < S; s += 32) cnt[s] = it.x0[traj * it.x0_stride + s];
            t = 0.0;
            xo_seed(g, it.seeds[traj]);
        }
        const double *rates = it.rate + traj * it.rate_stride;
        bool exact_traj = !spec_rate_ok((uint64_t)__double_as_longlong(t)) || !(t < 0x1p60);
        for (int r = lane; r < R; r += 32) exact_traj |= !spec_rate_ok((uint64_t)__double_as_longlong(rates[r]));
        if (!BATCH && it.rate_stride)
            for (int q = lane; q < 32 * C; q += 32) {
                const int r = (q & 31) * C + (q >> 5);
                const DF d = r < R ? df_from_double(rates[r]) : DF{0.f, 0.f};
                rdf_w[q] = make_float2(d.h, d.l);
            }
        exact_traj = __any_sync(0xffffffffu, exact_traj) || mm > 1024;  // (choice margins stay below 2^32 units)
        for (int s = lane; s <= S; s += 32) cntf[s] = s < S ? (float)cnt[s] : 1.0f;
        __syncwarp();
        unsigned long long ev = 0;

        // the generator before word q of the buffer that starts at state st
        auto state_at = [&](const uint64_t *st, int q) {
            Xoshiro h{st[0], st[1], st[2], st[3]};
            for (int k = 0; k < q; ++k) xo_next(h);
            return h;
        };
        for (long long i = 0; i < it.n_samples && !abort_run; ++i) {
            const double T = it.sample_t[i];
            // ---- interval start: save what an exact re-run needs
            for (int s = lane; s < S; s += 32) cnt0[s] = cnt[s];
            const int p0 = p;
            __syncwarp();
            if (lane == 0) {
                const bool empty = p == 32;  // then the generator itself is the state
                gst[8] = empty ? g.s0 : gst[0];
                gst[9] = empty ? g.s1 : gst[1];
                gst[10] = empty ? g.s2 : gst[2];
                gst[11] = empty ? g.s3 : gst[3];
            }
            const double t0 = t;
            const unsigned long long ev0 = ev;
            bool replay = exact_traj || !(T < 0x1p60) || (T != 0.0 && !(T >= 0x1p-60));
            // clock: units of 2^-et from t0 on; the interval (the sample time
            // itself when it is empty or lies behind t0) fills 2^50 .. 2^51
            const double len = __dsub_rn(T, t0);
            const double base = len > 0.0 ? len : (T > 0.0 ? T : 1.0);
            replay |= !(base >= 0x1p-60) || !(fabs(len) <= base * 0x1p2);
            const int et = replay ? 0 : 50 - ilog2d(base);
            const double ets = __longlong_as_double((long long)(1023 + et) << 52);
            const float etf = pow2f(et);
            const int64_t D = replay ? 0 : __double2ll_rn(__dmul_rn(len, ets));
            // what a step adds to the clock's error bound beside the quotient's:
            // the reference's rounding (2^-52 T), the conversions' units
            const int64_t err_step = replay ? 0 : __double2ll_ru(__dmul_ru(__dmul_ru(T, 0x1p-52), ets)) + 4;
            int64_t clk = 0, err = 2 * err_step;
            __syncwarp();
            unsigned int steps = 0;
            while (!replay) {
                if ((++steps & 255u) == 0) {
                    int late = lane == 0 && global_ns() - t_start > a.budget_ns;
                    if (__shfl_sync(0xffffffffu, late, 0)) {
                        abort_run = true;
                        break;
                    }
                }
                if (need_full || amb_next) {
                    // ---- every propensity of this lane's chunk, after the
                    // scale: 2^28 <= total * sc < 2^29
                    uint32_t mx = amb_next ? 0x7F800000u : 0u;
                    float mh = 0.0f, tf = 0.0f;
                    for (int i2 = 0; i2 < n_own && !amb_next; ++i2) {
                        float h = 0.0f;
                        eval_prop(i2 * 32 + lane, 1.0f, mx, h);
                        tf = __fadd_rn(tf, h);
                    }
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) tf = __fadd_rn(tf, __shfl_xor_sync(0xffffffffu, tf, d));
                    // an undecided step: a count out of range, a total beyond
                    // 2^90 or below 2^-90 (where a positive one is possible)
                    if (__any_sync(0xffffffffu, mx >= 0x4B000000u) || !(tf <= 0x1p90f) || (tf > 0.0f && tf < 0x1p-60f)) {
                        replay = true;
                        break;
                    }
                    absorbed = tf == 0.0f;
                    sc = absorbed ? 1.0f : pow2f(28 - ilog2f(tf));
                    ls = 0;
                    for (int i2 = 0; i2 < n_own; ++i2) {
                        const int64_t v = eval_prop(i2 * 32 + lane, sc, mx, mh);
                        prop[pz(i2 * 32 + lane)] = v;
                        ls += v;
                    }
                    need_full = false;
                    __syncwarp();
                }
                // ---- chunk prefixes and the total
                const int64_t incl = scan_i64(ls, 32);
                const int64_t tot = shfl_i64(incl, 31);
                if (tot < (1ll << 47)) {
                    if (absorbed) break;  // no reaction can fire: the sample records, no draw is made
                    need_full = true;     // too few bits left (a new scale's total has 50)
                    continue;
                }
                // ---- draws: refill the buffer when fewer than two words are left
                if (p > 30) {
                    __syncwarp();
                    int first = 0;
                    uint64_t w0 = 0;
                    if (p == 31) {  // the last word is still to come
                        first = 1;
                        w0 = (uint64_t)shfl_i64((int64_t)word, 31);
                        if (lane < 4) gst[lane] = gst[4 + lane];
                    } else if (lane == 0) {
                        gst[0] = g.s0;
                        gst[1] = g.s1;
                        gst[2] = g.s2;
                        gst[3] = g.s3;
                    }
                    word = w0;
                    for (int k = first; k < 31; ++k) {
                        const uint64_t w = xo_next(g);
                        if (lane == k) word = w;
                    }
                    __syncwarp();
                    if (lane == 0) {
                        gst[4] = g.s0;
                        gst[5] = g.s1;
                        gst[6] = g.s2;
                        gst[7] = g.s3;
                    }
                    const uint64_t w = xo_next(g);
                    if (lane == 31) word = w;
                    p = 0;
                    const int layer = (int)(word & 0xff);
                    const float2 X = xdf[layer];
                    x = df_mul(df_u53_rel(2 * (word >> 12) + 1), DF{X.x, X.y});
                    acc_mask = __ballot_sync(0xffffffffu, (word >> 12) < zxk[layer].y);
                    __syncwarp();
                }
                DF xe{__shfl_sync(0xffffffffu, x.h, p), __shfl_sync(0xffffffffu, x.l, p)};
                uint64_t bu = (uint64_t)shfl_i64((int64_t)word, p + 1);
                int used = p + 1;  // words consumed by the Exp1 draw, counted from the buffer's start
                const bool slow = !((acc_mask >> p) & 1u);
                Xoshiro gs{0, 0, 0, 0};
                if (slow) {
                    // wedge or tail (1.2 % of draws): the generator itself from
                    // here on, the buffer is given up
                    gs = state_at(gst, p);
                    xe = exp1_df_rel(gs, ex, xdf);
                }
                // ---- Exp1 / total in clock units, the decision
                const DF td = df_from_fx(tot);
                const DF q = df_div(xe, td, rcp_approx(td.h));  // / (sc 2^22)
                const float qh = fminf(__fmul_rn(__fmul_rn(q.h, sc), etf), 0x1p30f);
                const float ql = fmaxf(fminf(__fmul_rn(__fmul_rn(q.l, __fmul_rn(sc, 0x1p22f)), etf), 0x1p30f), -0x1p30f);
                const int64_t qc = fx_from_df(qh, ql);
                const int64_t clk_n = clk + qc;
                const int64_t err_n = err + err_step + (qc >> sh_q);
                const int64_t d = D - clk_n;
                if (d <= err_n || q.h < 0x1p-100f) {  // not a clear fire
                    if (d + err_n >= 0 || q.h < 0x1p-100f) {
                        replay = true;
                        break;
                    }
                    // the sample records; the Exp1 draw was made
                    if (slow) {
                        g = gs;
                        p = 32;
                    } else {
                        p = used;
                    }
                    break;
                }
                clk = clk_n;
                err = err_n;
                if (slow) {
                    bu = xo_next(gs);
                    g = gs;
                    p = 32;
                } else {
                    p = used + 1;
                }
                // ---- the choice: #{r : cum_r < total * U}
                const int64_t ch = (int64_t)__umul64hi((uint64_t)tot, bu & ~0x7FFull);
                const int64_t di = incl - ch;
                const int k = __popc(__ballot_sync(0xffffffffu, di < 0));  // chunks entirely below the choice
                const int64_t before = shfl_i64(incl - ls, k & 31);        // running sum before chunk k
                bool near = (uint32_t)((int)(di >> 32) + 1) <= 1u;         // |di| < 2^32
                // walk chunk k with the whole warp: lane j takes its reaction k*C + j
                int count = 0;
                int64_t carry = before - ch, dr = di;
                for (int seg = 0; seg < C; seg += 32) {
                    const int j = seg + lane;
                    const bool valid = j < C && k * C + j < R;
                    dr = carry + scan_i64(valid ? prop[pz(j * 32 + k)] : 0, C);
                    count += __popc(__ballot_sync(0xffffffffu, valid && dr < 0));
                    near |= (uint32_t)((int)(dr >> 32) + 1) <= 1u;
                    if (C > 32) carry = shfl_i64(dr, 31);
                }
                int idx = k * C + count;
                if (__any_sync(0xffffffffu, near) || a.exact_choice) {
                    // some sum lies within 2^32 units of the choice: within the
                    // margin the choice alone is redone exactly (the clock is
                    // decided; the fixed-point propensities are overwritten)
                    const int64_t m = (tot >> sh_p) + 4 * (int64_t)R + 16;
                    bool close = di <= m && di >= -m;
                    for (int seg = 0; seg < C; seg += 32) {
                        const int j = seg + lane;
                        if (seg == 0) carry = before - ch;
                        dr = carry + scan_i64(j < C && k * C + j < R ? prop[pz(j * 32 + k)] : 0, 32);
                        close |= dr <= m && dr >= -m;
                        carry = shfl_i64(dr, 31);
                    }
                    if (__any_sync(0xffffffffu, close) || a.exact_choice) {
                        __syncwarp();
                        idx = warp_exact_choice<MACRO>(it, cnt, rates, scr, bu >> 11);
                        need_full = true;
                    }
                }
                // ---- jump
                ++ev;
                if (idx < R)
                    for (int q2 = lane; q2 < Q; q2 += 32) {
                        int sp;
                        int64_t dlt;
                        if (BATCH || jd_wide) {
                            sp = it.jmp_sp[idx * Q + q2];
                            dlt = it.jmp_d[idx * Q + q2];
                        } else {
                            const uint32_t e = jump_sh[idx * Q + q2];
                            sp = (int)(e & 0xFFFFu);
                            dlt = (int64_t)((int32_t)e >> 16);
                        }
                        if (dlt != 0) {
                            cnt[sp] += dlt;
                            cntf[sp] = __fadd_rn(cntf[sp], (float)dlt);
                        }
                    }
                __syncwarp();
                // ---- re-evaluate this lane's propensities that read a changed
                // species; their differences go to the chunk sum
                if (idx < R && !need_full) {
                    uint32_t mx = 0u;
                    float mh = 0.0f;
                    for (int w = 0; w < n_words; ++w) {
                        const size_t e = ((size_t)idx * n_words + w) * 32 + lane;
                        const int left = n_own - 32 * w;
                        uint32_t m = left >= 32 ? 0xFFFFFFFFu : left > 0 ? (1u << left) - 1u : 0u;
                        if (dep_tab)
                            m = dep_bytes == 1   ? reinterpret_cast<const uint8_t *>(dep_tab)[e]
                                : dep_bytes == 2 ? reinterpret_cast<const uint16_t *>(dep_tab)[e]
                                                 : reinterpret_cast<const uint32_t *>(dep_tab)[e];
                        while (m) {
                            const int pos = (32 * w + __ffs((int)m) - 1) * 32 + lane;
                            m &= m - 1u;
                            const int64_t v = eval_prop(pos, sc, mx, mh);
                            const int ps = pz(pos);
                            ls += v - prop[ps];
                            prop[ps] = v;
                        }
                    }
                    __syncwarp();
                    // a count out of range makes the next step undecided, a
                    // sum that outgrew the fixed point asks for a new scale
                    const bool out = mx >= 0x4B000000u;
                    if (__any_sync(0xffffffffu, out || !(mh < 0x1p30f) || (uint64_t)ls >> kFxLim != 0)) {
                        amb_next = __any_sync(0xffffffffu, out);
                        need_full = true;
                    }
                }
            }
            if (abort_run) break;
            if (replay) {
                // ---- exact re-run of the interval from its saved start
                if (!exact_traj && lane == 0) atomicAdd(a.work + 3, 1ull);
                for (int s = lane; s < S; s += 32) cnt[s] = cnt0[s];
                g = state_at(gst + 8, p0 == 32 ? 0 : p0);
                p = 32;
                t = t0;
                ev = ev0;
                __syncwarp();
                for (unsigned int n = 1;; ++n) {
                    if ((n & 255u) == 0) {
                        int late = lane == 0 && global_ns() - t_start > a.budget_ns;
                        if (__shfl_sync(0xffffffffu, late, 0)) {
                            abort_run = true;
                            break;
                        }
                    }
                    int idx = 0;
                    if (!warp_exact_step<MACRO>(it, cnt, rates, a.zig, scr, g, t, T, idx)) break;
                    ++ev;
                    if (idx < R)
                        for (int q = lane; q < Q; q += 32) {
                            const int64_t dlt = it.jmp_d[idx * Q + q];
                            if (dlt != 0) cnt[it.jmp_sp[idx * Q + q]] += dlt;
                        }
                    __syncwarp();
                }
                if (abort_run) break;
                for (int s = lane; s < S; s += 32) cntf[s] = (float)cnt[s];
                need_full = true;
                amb_next = false;
                // lane 0 drew: its generator is the trajectory's
                g.s0 = (uint64_t)shfl_i64((int64_t)g.s0, 0);
                g.s1 = (uint64_t)shfl_i64((int64_t)g.s1, 0);
                g.s2 = (uint64_t)shfl_i64((int64_t)g.s2, 0);
                g.s3 = (uint64_t)shfl_i64((int64_t)g.s3, 0);
                __syncwarp();
            }
            // ---- record sample i at t = T
            t = T;
            int64_t *o = it.out + (size_t)i * it.n_save * it.n_traj + traj;
            for (int k = lane; k < it.n_save; k += 32) o[(size_t)k * it.n_traj] = cnt[it.save_idx[k]];
            __syncwarp();
        }
        if (abort_run) {
            if (lane == 0) atomicExch(a.work + 2, 1ull);
            break;
        }
        if (it.fin_species)
            for (int s = lane; s < S; s += 32) it.fin_species[traj * S + s] = cnt[s];
        if (it.fin_rng && p < 32) g = state_at(gst, p);
        if (lane == 0) {
            if (it.fin_t) it.fin_t[traj] = t;
            if (it.fin_rng) {
                it.fin_rng[traj * 4 + 0] = g.s0;
                it.fin_rng[traj * 4 + 1] = g.s1;
                it.fin_rng[traj * 4 + 2] = g.s2;
                it.fin_rng[traj * 4 + 3] = g.s3;
            }
            if (it.events) it.events[traj] = ev;
        }
        warp_events += ev;
        __syncwarp();
    }
    if (lane == 0 && warp_events) atomicAdd(a.work + 1, warp_events);
}

template <bool MACRO, bool BATCH>
int warp_launch(const SsaArgs &a, int block, int grid, size_t smem, cudaStream_t st) {
    auto kern = ssa_warp_kernel<MACRO, BATCH>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    kern<<<grid, block, smem, st>>>(a);
    return (int)cudaGetLastError();
}

}  // namespace

int ssa_warp_warps(const SsaArgs &a, size_t smem_limit) {
    const WarpLayout l = warp_layout(a);
    if (l.block_bytes + l.warp_bytes > smem_limit) return 0;
    return (int)std::min<size_t>(a.batch ? kWarpMaxWarpsBatch : kWarpMaxWarps, (smem_limit - l.block_bytes) / l.warp_bytes);
}

size_t ssa_warp_smem(const SsaArgs &a, int warps) {
    const WarpLayout l = warp_layout(a);
    return l.block_bytes + (size_t)warps * l.warp_bytes;
}

bool ssa_warp_supported(const SsaArgs &a, int max_order) {
    return a.ex_off == nullptr && a.S < 65536 && max_order < 32768 && a.R >= 1;
}

int ssa_warp_occupancy(const SsaArgs &a, int warps, size_t smem) {
    int n = 0;
    // the arithmetic variants share the block shape and shared memory use;
    // batch launches have their own register budget
    const auto k = a.batch ? ssa_warp_kernel<false, true> : ssa_warp_kernel<false, false>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * warps, smem);
    return n;
}

int launch_ssa_warp(const SsaArgs &a, int warps, int grid, size_t smem, void *stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool batch = a.batch != nullptr;
    if (a.macro_mode)
        return batch ? warp_launch<true, true>(a, 32 * warps, grid, smem, st)
                     : warp_launch<true, false>(a, 32 * warps, grid, smem, st);
    return batch ? warp_launch<false, true>(a, 32 * warps, grid, smem, st)
                 : warp_launch<false, false>(a, 32 * warps, grid, smem, st);
}

uint32_t warp_shape_word(const int32_t *fac_sp, const int32_t *fac_ord, int P, int S, int r) {
    return shape_word(fac_sp, fac_ord, P, S, r);
}

}  // namespace rbg
