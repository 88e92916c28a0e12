// mbarrier and TMA (cp.async.bulk.tensor) helpers shared by the kernels that stage operands with TMA.
//
// Every wait is bounded: `mbar_wait` polls at most WAIT_LIMIT times and then returns false; the caller records
// OXR_WAIT_EXPIRED in the status word, stops waiting, releases what it holds and returns, so a kernel can never hang
// on a barrier that nobody completes.
#pragma once

#include <cuda.h>

#include "common.cuh"

constexpr uint32_t WAIT_LIMIT = 1u << 22;   // polls of an mbarrier before giving up (seconds at most)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Poll until the phase with the given parity has completed. False if the limit of polls ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_addr(bar);
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// One tile of a 2-D tensor map into shared memory; c0 is the innermost coordinate (its byte offset must be a
// multiple of 16), c1 the row. Completion is counted in bytes on `bar`. No multicast.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(c0), "r"(c1) : "memory");
}
// One box of a 3-D tensor map (c0 innermost, its byte offset a multiple of 16).
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// Orders earlier ordinary shared-memory accesses, reads too, before later accesses by TMA or bulk copies to the same addresses.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// A warp has read its part of a stage with ordinary loads, and the stage may be filled again. Without the fence the arrival did not wait for reads still on their
// way: where a decode step's products started behind an attention kernel, the next slice's copy landed under a warp's last 64 bytes of a weight row.
__device__ __forceinline__ void mbar_release_stage(uint64_t* bar, int lane) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// ---------------------------------------------------------------------------------------------------- host side
typedef CUresult (*OxrEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                     const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                     CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline OxrEncodeTiledFn oxr_encode_tiled() {
    static OxrEncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<OxrEncodeTiledFn>(p);
    }
    return fn;
}

// A [rows, cols] bf16 row-major matrix seen as tiles of box_rows x 64 columns (128 bytes), 128-byte swizzle;
// elements outside the matrix read as zero. cols must be a multiple of 8 (rows are whole 16-byte words).
static inline bool oxr_make_map_bf16(CUtensorMap* map, const void* base, unsigned long long rows, unsigned long long cols, int box_rows) {
    OxrEncodeTiledFn fn = oxr_encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A [tokens, heads, d] bf16 tensor (contiguous) seen as boxes of box_tokens x box_heads x 64 d (128 bytes), 128-byte swizzle:
// a box lands as rows of 128 bytes in the order (token, head). Elements outside the tensor read as zero.
static inline bool oxr_make_map_bf16_3d(CUtensorMap* map, const void* base, unsigned long long tokens, unsigned long long heads,
                                        unsigned long long d, int box_tokens, int box_heads) {
    OxrEncodeTiledFn fn = oxr_encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)tokens};
    const cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)d * heads * 2};
    const cuuint32_t box[3] = {64u, (cuuint32_t)box_heads, (cuuint32_t)box_tokens};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
