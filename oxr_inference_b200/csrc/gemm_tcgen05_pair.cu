// bf16 GEMM on the 5th-generation tensor cores with two SMs per tile: C[M,N] = X[M,K] * W[N,K]^T for many rows.
//
// The reference multiplies through nn.Linear / cuBLAS (oxr_runtime/language.py:223-244,261,268-269). The one-SM
// kernel fills 16 KB of X and up to 32 KB of W into shared memory per 64-wide k step of a 128 x 256 tile; with a
// third less to fill per block the tensor pipe waits less (a k step measured 0.42 us per block instead of 0.45 us).
// Two blocks of a cluster share a 256 x bn tile (tcgen05 cta_group::2):
//   * block r of the pair stages rows 128 r .. + 127 of the X tile and rows bn/2 r .. of the W tile, by TMA, STAGES
//     deep: per k step half the W bytes of the one-SM kernel for the same 128 x bn of output per block;
//   * the pair's leader (rank 0) issues tcgen05.mma.cta_group::2 with M = 256, N = bn: the tensor cores of both SMs
//     read X from their own shared memory and the halves of W from both, and accumulate 128 x bn each in their own
//     tensor memory;
//   * the barriers that count TMA bytes live in the leader (both blocks' copies complete on them), tcgen05.commit
//     with a cluster mask frees a stage in both blocks and hands the accumulator to both blocks' epilogue warps,
//     which give it back by arriving on the leader's barrier;
//   * tiles are walked persistently by the pairs, two accumulators in tensor memory overlap epilogue and MMA.
// ACROSS has W along the 256-row side of the tile and the rows of X as its width, any multiple of 32: the same products transposed, for numbers of rows that fill
// tiles of 256 badly (1,562 rows x 24,576 x 4,096 gated 262 us in 7 x 256 rows, 226 in 10 x 160; 1,421 x 4,096 x 12,288 135 and 112). Its epilogue costs 4 to 9 us
// a product more (the accumulator comes out column by column), so where the rows do fill the tiles the plain form stays.
// No TMA copy is multicast. Every wait on an mbarrier is bounded as in the one-SM kernel; both blocks meet at a
// cluster barrier before tensor memory is freed, so neither leaves while the other may still touch its memory.
#include "umma.cuh"

namespace {
constexpr int PAIR_THREADS = 192;   // warp 0: TMA, warp 1: MMA (leader) + TMEM owner, warps 2..5: epilogue

__host__ __device__ constexpr int pair_stage_bytes(int bn) { return A_BYTES + (bn / 2) * BK * 2; }

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The address, in the cluster's shared window, of the same shared-memory location in block `rank` of the cluster.
__device__ __forceinline__ uint32_t in_block(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA tile load whose bytes are counted on a barrier that may live in the pair's other block (cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void umma_pair_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on the barrier at this shared-memory offset in both blocks of the pair when the MMAs issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_addr(bar)), "h"((uint16_t)3) : "memory");
}

struct PairTile { int m0, n0; };   // rows of X from m0, rows of W from n0

// Tile order as in the one-SM kernel, with 256-row tiles: pairs that run at the same time share few W tiles. ACROSS: tiles of 256 rows of W by
// bn rows of X, all tiles of rows of X for one W tile and then the next.
template <bool ACROSS>
__device__ __forceinline__ PairTile pair_tile(int tile, int M, int N, int bn) {
    if constexpr (ACROSS) {
        const int tiles_x = (M + bn - 1) / bn;
        return {tile % tiles_x * bn, tile / tiles_x * 2 * BM};
    }
    constexpr int GROUP_M = 16;
    const int tiles_m = (M + 2 * BM - 1) / (2 * BM), tiles_n = (N + bn - 1) / bn;
    const int per_group = GROUP_M * tiles_n;
    const int group = tile / per_group, within = tile % per_group;
    const int group_rows = min(GROUP_M, tiles_m - group * GROUP_M);
    return {(group * GROUP_M + within % group_rows) * 2 * BM, (within / group_rows) * bn};
}

// ACROSS: the four epilogue warps of a block have a column of C per lane, 128 in all, and turn a piece of up to 32 rows over in shared memory: rows of 128 columns
// (GATED 64) and 16 bytes against bank conflicts, which then leave in whole 16-byte words, 256 (128) bytes of a row side by side. (Stored from the registers, two bytes
// a lane and 32 or 64 bytes of a row at a time, a gated product of 1,562 x 24,576 x 4,096 in tiles of 160 took 317 us instead of 226.)
template <typename TO, bool GATED> struct Turned {
    static constexpr int COLS = GATED ? 64 : 128, PITCH = COLS * (int)sizeof(TO) + 16, BYTES = 2 * 32 * PITCH;   // two pieces: one barrier each
};
template <typename TO, bool GATED>
__device__ __forceinline__ void turn_piece(unsigned char* buf, const uint32_t (&v)[32], int count, int col, const GateForm& gate) {   // col: 0 .. 127
    using T = Turned<TO, GATED>;
    if constexpr (!GATED) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < count) *reinterpret_cast<TO*>(buf + j * T::PITCH + col * (int)sizeof(TO)) = Num<TO>::from_f32(__uint_as_float(v[j]));
    } else {
        // gate and up columns alternate in eights: lanes 0..7 and 16..23 have gates, the lanes eight behind them their ups. A gate's lane keeps every even row and gets
        // its up, an up's lane gets the gates of the odd ones.
        const bool up = col & 8;
        TO* at = reinterpret_cast<TO*>(buf + (up ? T::PITCH : 0)) + col / 16 * 8 + col % 8;
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            const float mine = __uint_as_float(up ? v[j + 1] : v[j]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? v[j] : v[j + 1]), 8);
            if (j < count) *reinterpret_cast<TO*>(reinterpret_cast<unsigned char*>(at) + j * T::PITCH) = Num<TO>::from_f32(gate_apply(gate, up ? other : mine, up ? mine : other));
        }
    }
}
// rows row0 .. of C, columns from col0 on, `width` columns of C in all
template <typename TO, bool GATED>
__device__ __forceinline__ void store_turned(TO* __restrict__ C, const unsigned char* buf, int rows, int row0, int col0, int width) {
    using T = Turned<TO, GATED>;
    constexpr int PER = 16 / (int)sizeof(TO), WORDS = T::COLS / PER;
    const bool whole = width % PER == 0 && (uintptr_t)C % 16 == 0;
    for (int i = threadIdx.x - 64; i < rows * WORDS; i += 128) {
        const int r = i / WORDS, c = i % WORDS * PER;
        if (col0 + c >= width) continue;
        const uint4 word = *reinterpret_cast<const uint4*>(buf + r * T::PITCH + c * (int)sizeof(TO));
        TO* at = C + (size_t)(row0 + r) * width + col0 + c;
        if (whole) *reinterpret_cast<uint4*>(at) = word;
        else {
            const TO* e = reinterpret_cast<const TO*>(&word);
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (col0 + c + k < width) at[k] = e[k];
        }
    }
}
// Barrier 1 is the epilogue warps' own (128 threads).
__device__ __forceinline__ void turn_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ bool turn_all(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.and.pred p, 1, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r) : "r"((uint32_t)v) : "memory");
    return r != 0;
}

template <typename TO, bool GATED, bool ACROSS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_pair_kernel(TO* __restrict__ C, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                         int M, int N, int K, int bn, int stages, int tmem_cols, int num_tiles, int* status, const GateForm gate) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // swizzle atoms are 1024 B
    const int stage_size = pair_stage_bytes(bn);
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)stages * stage_size);   // used in the leader only
    uint64_t* empty = full + MAX_STAGES;
    uint64_t* accum_full = empty + MAX_STAGES;   // [2] MMA -> epilogue, in each block
    uint64_t* accum_empty = accum_full + 2;      // [2] epilogue -> MMA, used in the leader only: 8 arrivals (4 warps x 2 blocks)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum_empty + 2);
    uint32_t* gave_up = tmem_slot + 1;
    static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= BARRIER_BYTES, "barriers outgrow their space");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int num_kb = (K + BK - 1) / BK;
    const uint32_t acc_stride = (uint32_t)tmem_cols / 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(accum_full + i, 1); mbar_init(accum_empty + i, 8); }
        *gave_up = 0;
        mbar_fence_init();
    }
    if (warp == 1) {   // one warp of each block of the pair: the allocation is made in both blocks' tensor memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"((uint32_t)tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();   // both blocks' barriers are initialised before either signals the other's
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (each block its halves)
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            // No kernel writes the weights: this block's halves of W's tiles for the first ring of stages are requested
            // before the kernel (when it is launched dependent on the one before) waits for that one; the rows of X for
            // the same stages follow after the wait. The leader arms each of these stages for both blocks' bytes.
            auto load_w = [&](int stage, int kb, const PairTile& t, uint32_t bar) {
                unsigned char* dst = tiles + (size_t)stage * stage_size;
                if constexpr (ACROSS) tma_load_2d_pair(dst, &map_w, kb * BK, t.n0 + (int)rank * BM, bar);
                else tma_load_2d_pair(dst + A_BYTES, &map_w, kb * BK, t.n0 + (int)rank * (bn / 2), bar);
            };
            auto load_x = [&](int stage, int kb, const PairTile& t, uint32_t bar) {
                unsigned char* dst = tiles + (size_t)stage * stage_size;
                if constexpr (ACROSS) tma_load_2d_pair(dst + A_BYTES, &map_x, kb * BK, t.m0 + (int)rank * (bn / 2), bar);
                else tma_load_2d_pair(dst, &map_x, kb * BK, t.m0 + (int)rank * BM, bar);
            };
            int early = 0;
            for (int tile = pair; tile < num_tiles && early < stages; tile += num_pairs) {
                const PairTile t = pair_tile<ACROSS>(tile, M, N, bn);
                for (int kb = 0; kb < num_kb && early < stages; ++kb, ++early) {
                    if (rank == 0) mbar_expect_tx(full + early, 2u * (uint32_t)stage_size);
                    load_w(early, kb, t, in_block(smem_addr(full + early), 0));
                }
            }
            pdl_wait();
            int step = 0;
            for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
                const PairTile t = pair_tile<ACROSS>(tile, M, N, bn);
                for (int kb = 0; kb < num_kb; ++kb, ++step) {
                    const uint32_t leader_full = in_block(smem_addr(full + s), 0);
                    if (step < early) {   // first ring: the stage is free and armed, its part of W's tile is on its way
                        load_x(s, kb, t, leader_full);
                    } else {
                        if (!mbar_wait(empty + s, phase ^ 1)) { atomicExch(gave_up, 1u); oxr_report(status, OXR_WAIT_EXPIRED, 10); ok = false; break; }
                        if (rank == 0) mbar_expect_tx(full + s, 2u * (uint32_t)stage_size);   // both blocks' bytes
                        load_x(s, kb, t, leader_full);
                        load_w(s, kb, t, leader_full);
                    }
                    if (++s == stages) { s = 0; phase ^= 1; }
                }
            }
            pdl_trigger();   // every load of this block is issued: a chained kernel after this one may be scheduled
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (the leader's one thread)
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc(2 * BM, bn);
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            int it = 0;
            for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++it) {
                const int acc = it & 1;
                const uint32_t acc_phase = (it >> 1) & 1;
                if (!mbar_wait(accum_empty + acc, acc_phase ^ 1)) { atomicExch(gave_up, 1u); oxr_report(status, OXR_WAIT_EXPIRED, 13); ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmem_d = tmem_base + (uint32_t)acc * acc_stride;
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait(full + s, phase)) { atomicExch(gave_up, 1u); oxr_report(status, OXR_WAIT_EXPIRED, 11); ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_addr = smem_addr(tiles + (size_t)s * stage_size);
                    const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma_pair_bf16(tmem_d, umma_desc(a_addr + k * UMMA_K * 2), umma_desc(b_addr + k * UMMA_K * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(empty + s);   // the stage is free in both blocks once these MMAs have read it
                    if (++s == stages) { s = 0; phase ^= 1; }
                }
                umma_commit_pair(accum_full + acc);   // both blocks' epilogues may read (also after giving up)
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: this block's 128 rows
        pdl_wait();   // C may still be read by the kernels before this one
        const int quarter = warp & 3;
        [[maybe_unused]] unsigned char* turned = reinterpret_cast<unsigned char*>(full) + BARRIER_BYTES;
        [[maybe_unused]] int piece = 0;
        int it = 0;
        for (int tile = pair; tile < num_tiles; tile += num_pairs, ++it) {
            const PairTile t = pair_tile<ACROSS>(tile, M, N, bn);
            const int acc = it & 1;
            const uint32_t acc_phase = (it >> 1) & 1;
            [[maybe_unused]] const int row = t.m0 + (int)rank * BM + quarter * 32 + lane;
            bool ok = mbar_wait(accum_full + acc, acc_phase);
            if (!ok) { atomicExch(gave_up, 1u); if (lane == 0) oxr_report(status, OXR_WAIT_EXPIRED, 12); }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            ok = ok && (*reinterpret_cast<volatile uint32_t*>(gave_up) == 0);
            if constexpr (ACROSS) ok = turn_all(ok);          // the four warps meet at barriers below: they leave together
            else ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t acc_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * acc_stride;
#pragma unroll 1
            for (int c0 = 0; c0 < bn; c0 += 32) {
                uint32_t v[32];
                const int count = min(32, bn - c0);
                if (count == 32) tmem_ld_32x32(acc_addr + (uint32_t)c0, v);
                else tmem_ld_32x16(acc_addr + (uint32_t)c0, v);
                if constexpr (ACROSS) {
                    unsigned char* buf = turned + (piece & 1) * 32 * Turned<TO, GATED>::PITCH;   // last read before the barrier of the piece between
                    ++piece;
                    if (!GATED && gate.kind == 2) relu2_piece(v);
                    turn_piece<TO, GATED>(buf, v, count, quarter * 32 + lane, gate);
                    turn_sync();
                    const int col0 = t.n0 + (int)rank * BM;
                    store_turned<TO, GATED>(C, buf, min(count, M - t.m0 - c0), t.m0 + c0, GATED ? col0 / 2 : col0, GATED ? N / 2 : N);
                } else if (row < M && t.n0 + c0 < N) {
                    if constexpr (GATED) store_row_piece_gated<TO>(C + (size_t)row * (N / 2) + (t.n0 + c0) / 2, v, count, t.n0 + c0, N, gate);
                    else {
                        if (gate.kind == 2) relu2_piece(v);   // the plain product's optional activation
                        store_row_piece<TO>(C + (size_t)row * N + t.n0 + c0, v, count, t.n0 + c0, N);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_block(smem_addr(accum_empty + acc), 0));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();   // neither block frees or leaves while the other may still read its shared or tensor memory
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)tmem_cols) : "memory");
    }
}

template <typename TO, bool GATED, bool ACROSS>
int launch_pair(void* C, const void* X, const void* W, int M, int N, int K, int bn, int* status, cudaStream_t stream, int act = 0) {
    static int max_pairs = 0;   // per instantiation
    if (max_pairs == 0) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<TO, GATED, ACROSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return 1000 + (int)e;
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 2) sms = 148;
        // how many pairs the device holds at once: ask, and fall back to one per two SMs
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
        cfg.blockDim = dim3(PAIR_THREADS);
        cfg.dynamicSmemBytes = SMEM_BYTES;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, gemm_tcgen05_pair_kernel<TO, GATED, ACROSS>, &cfg) != cudaSuccess || clusters <= 0) {
            (void)cudaGetLastError();
            clusters = sms / 2;
        }
        max_pairs = clusters < sms / 2 ? clusters : sms / 2;
    }
    CUtensorMap map_x, map_w;
    if (!oxr_make_map_bf16(&map_x, X, M, K, ACROSS ? bn / 2 : BM) || !oxr_make_map_bf16(&map_w, W, N, K, ACROSS ? BM : bn / 2)) return OXR_BAD_ARGUMENT;
    const long long tiles = ACROSS ? (long long)((N + 2 * BM - 1) / (2 * BM)) * ((M + bn - 1) / bn) : (long long)((N + bn - 1) / bn) * ((M + 2 * BM - 1) / (2 * BM));
    if (tiles > 0x7fffffffLL) return OXR_BAD_ARGUMENT;
    int stages = (RING_BYTES - (ACROSS ? Turned<TO, GATED>::BYTES : 0)) / pair_stage_bytes(bn);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    int tmem_cols = 32;
    while (tmem_cols < 2 * bn) tmem_cols *= 2;
    const unsigned pairs = (unsigned)(tiles < max_pairs ? tiles : max_pairs);
    oxr_launch(gemm_tcgen05_pair_kernel<TO, GATED, ACROSS>, dim3(2 * pairs), dim3(PAIR_THREADS), SMEM_BYTES, stream, true, (TO*)C, map_x, map_w, M, N, K,
               bn, stages, tmem_cols, (int)tiles, status, act == 1 ? RELU2_FORM : (GATED ? oxr_gate_form : PLAIN_FORM));
    return oxr_launch_status();
}
}  // namespace

// out_dtype: 0 = float32, 1 = bfloat16. Requires K % 8 == 0 and 16-byte aligned X, W. tile: the size, a multiple of 32 from 32 to 256, of a pair's tile along
// the side that is not 256 long: columns of the output (each block stages half of them), or, with `across`, rows. act 1: the output is relu(x)^2 of the fp32 sums.
OXR_API int oxr_gemm_tcgen05_pair_bf16(void* C, const void* X, const void* W, int M, int N, int K, int out_dtype, int tile, int across, int act, int* status,
                                       cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (act != 0 && act != 1) return OXR_BAD_ARGUMENT;
    if (K <= 0 || K % 8 != 0 || (uintptr_t)X % 16 != 0 || (uintptr_t)W % 16 != 0) return OXR_BAD_ARGUMENT;
    if (tile < 32 || tile > MAX_BN || tile % 32 != 0) return OXR_BAD_ARGUMENT;
    if (out_dtype == 1 && across) return launch_pair<__nv_bfloat16, false, true>(C, X, W, M, N, K, tile, status, stream, act);
    if (out_dtype == 1) return launch_pair<__nv_bfloat16, false, false>(C, X, W, M, N, K, tile, status, stream, act);
    if (out_dtype == 0 && across) return launch_pair<float, false, true>(C, X, W, M, N, K, tile, status, stream, act);
    if (out_dtype == 0) return launch_pair<float, false, false>(C, X, W, M, N, K, tile, status, stream, act);
    return OXR_BAD_ARGUMENT;
}

// C [M, N / 2] = silu(X Wg^T) * (X Wu^T) in bf16 for W [N, K] whose gate and up rows alternate in groups of 8 (N a
// multiple of 16): the pair kernel with the gated epilogue.
OXR_API int oxr_gemm_tcgen05_pair_gated_bf16(void* C, const void* X, const void* W, int M, int N, int K, int tile, int across, int* status,
                                             cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (N % 16 != 0 || K <= 0 || K % 8 != 0 || (uintptr_t)X % 16 != 0 || (uintptr_t)W % 16 != 0 || (uintptr_t)C % 16 != 0) return OXR_BAD_ARGUMENT;
    if (tile < 32 || tile > MAX_BN || tile % 32 != 0) return OXR_BAD_ARGUMENT;
    if (across) return launch_pair<__nv_bfloat16, true, true>(C, X, W, M, N, K, tile, status, stream);
    return launch_pair<__nv_bfloat16, true, false>(C, X, W, M, N, K, tile, status, stream);
}
