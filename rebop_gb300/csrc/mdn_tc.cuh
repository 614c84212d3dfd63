// Pieces shared by the surrogate's tensor-core kernels (mdn.cu, mdn_train.cu):
// tcgen05 operand descriptors, TMA loads and tensor maps, the head's layout.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <utility>
#include <vector>

namespace rbg {

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

constexpr int kTmM = 128, kTmN = 64, kTmK = 64, kTmStages = 4;
constexpr int kTmABytes = kTmM * kTmK * 2, kTmBBytes = kTmN * kTmK * 2, kTmStage = kTmABytes + kTmBBytes;
constexpr size_t kTmSmem = (size_t)kTmStages * kTmStage + 1024;  // + alignment slack to 1 KiB

// Shared-memory descriptor of a K-major operand in the 128-byte swizzle:
// stride between 8-row atoms 1024 B, leading offset unused (1), version 1,
// layout type 2 (128-byte swizzle) in bits 61-63.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + __expf(-x)); }

__device__ __forceinline__ float softplusf_(float x) { return x > 20.0f ? x : log1pf(__expf(x)); }


// Count-aware head: classes per species (the last one the tail's), at most
// kKTMax tail components.
constexpr int kNC = 32, kKTMax = 16;


}  // namespace

}  // namespace rbg

namespace {

// Dynamic shared memory above 48 KB for `kern`, asked once per (kernel, device):
// the attribute belongs to the current device's context.
cudaError_t opt_in_smem(const void *kern, size_t bytes) {
    static std::mutex mu;
    static std::vector<std::pair<const void *, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    for (const auto &d : done)
        if (d.first == kern && d.second == dev) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done.emplace_back(kern, dev);
    return e;
}

// 2-D tensor map of a row-major BF16 matrix [rows][K] (row pitch ld elements)
// read in boxes of 64 (K) x box_rows with the 128-byte swizzle; false if the
// driver has no encoder or refuses the operands.
bool encode_rows(CUtensorMap &map, const void *base, int rows, int K, int ld, int box_rows) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    if (!encode) return false;
    const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t stride[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)rbg::kTmK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dim, stride, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}


}  // namespace
