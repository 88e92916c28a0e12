// 32-bit GEMM: C[M,N] = A[M,K] * W[N,K]^T on the bf16 tensor cores, in parts of eight bits (no TF32). Short rows: gemm_f32_short.cu.
//
// This is the matrix product of the 32-bit path of the whole model (the reference multiplies through
// nn.Linear, oxr_runtime/language.py:223-244; in fp32 only on the CPU in its tests).
//
// A 24-bit significand is three of 8 bits (the split into bf16 parts is that of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations", 2019): x = x0 + x1 + x2, each part x less the parts before it, rounded to bf16. Both operands are first multiplied by 2^16 and their
// sums by 2^-32: bf16's smallest number is then fp32's, 2^-149, and the parts of every fp32 number add up to it exactly, those of the smallest too
// (unscaled, a third part fell out of bf16's range below 2^-108, and operands of 2^-126 kept 9 bits). Products of two parts are exact in fp32, so a product of A and W is
// w0 a0 + (w0 a1 + w1 a0) + (w0 a2 + w1 a1 + w2 a0) up to 2^-24 of it (w1 a2, w2 a1 and w2 a2 are left out), and a W whose values are bf16 numbers, as a widened checkpoint's are, has
// w1 = w2 = 0: three products, exact. Sums: over each chunk of 64 k the head products w0 a0 go into one accumulator in tensor memory and the others into a second one;
// the two are added, and then to a sum in registers, rounded to nearest; K / 1,024 segments of k, one at least and four at most, of whole chunks (the last is shorter), have
// a sum each, and these are added in order. So an element's result depends on its row and column alone, not on M, the tile, or how the work is dealt out.
// Error of an element: 16 + K / 64 times 2^-24 of the magnitudes' sum at most (a chunk's sixteen-term sums inside the tensor core lose up to 2^-23 of what is there, K / 64 + 4
// roundings follow), where K fused multiply-adds one after the other allow K times 2^-24.
//
// Two kernels. `split_rows_kernel` writes A's parts, [3][M][K] in bf16. `gemm_f32_kernel` has W on the 128-row side of the tcgen05 tile
// (split on the way from global to shared memory) and the rows of A as the tile's width, any multiple of 16, so that a trace's few hundred rows waste none.
// Measured (2-norms against 64 bits, normal inputs, and of K fused multiply-adds in the order of k): K = 128 7.5e-8 and 2.0e-7, 1,024 1.0e-7 and 5.7e-7, 2,048 1.1e-7 and 8.1e-7,
// 8,192 1.3e-7 and 1.6e-6; all positive 128 9.0e-8 and 1.8e-7, 2,048 9.6e-8 and 7.0e-7.
// What bounds it: a chunk's way through a block, 1.0 us and 0.006 for each row of the tile: the issuing thread's waits, W's trip to the splitters and the adders' reads
// of tensor memory, eight columns at a time for want of registers; its products take 0.4 us. 333 rows, a graph of products with other weights each, against 8 x 8 register
// tiles of fused multiply-adds (42 TFLOP/s at best): 3,072 x 2,048 31 us (124), 2,048 x 2,048 29 (107), 16,384 x 2,048 169 (527), 2,048 x 8,192 88 (431); 40 rows 16,384 x
// 2,048 57 (117); one row 16,384 x 2,048 51 (330), 3,072 x 2,048 24 (316); 2,048 rows 16,384 x 2,048 776 (2,609), 2,048 x 8,192 413 (1,532). A W of 24-bit numbers takes six
// products and a full split: 333 rows 41, 39, 223 and 125 us in the order above, one row 63 and 31, 2,048 rows 1,044 and 556.
#include "umma.cuh"

namespace {
constexpr int F32_CHUNK = 64;          // k per accumulator: one 128-byte row of bf16
constexpr int F32_ADDERS = 8, F32_WORKERS = 16;   // warps 0..7 add the accumulators up, 8..15 split W
constexpr int F32_THREADS = (F32_WORKERS + 2) * 32;
constexpr int F32_W_PART = 128 * F32_CHUNK * 2, F32_W_STAGE = 3 * F32_W_PART;
constexpr int F32_AHEAD = 8;           // chunks that one prefetch of a row of W covers (2 KB: 6 to 10 % faster than none, 4 chunks in between)
constexpr int F32_CHUNKS = 8;          // chunks with barriers of their own
constexpr int F32_MAX_TILE = 128, F32_MAX_SLOTS = 8, F32_MAX_SEGMENTS = 4, F32_MIN_SEGMENT = 1024;

struct Parts { uint32_t p0, p1, p2; };     // two neighbouring values' parts, packed

constexpr float F32_SCALE = 65536.f, F32_UNSCALE = 0x1p-32f;     // what both operands are multiplied by, and their sums

__device__ __forceinline__ uint32_t bits2(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }

// F32_SCALE v = hi + mid + lo. An infinite hi (also one that a finite v makes, from 2^111 on) or a NaN stands alone: the epilogue sees to such results.
__device__ __forceinline__ Parts split2(float a, float b) {
    Parts r;
    a *= F32_SCALE;
    b *= F32_SCALE;
    r.p0 = bits2(__floats2bfloat162_rn(a, b));
    const float a0 = __uint_as_float(r.p0 << 16), b0 = __uint_as_float(r.p0 & 0xffff0000u);
    float a1 = a - a0, b1 = b - b0;
    if ((r.p0 & 0x7f80u) == 0x7f80u) a1 = 0.f;
    if ((r.p0 & 0x7f800000u) == 0x7f800000u) b1 = 0.f;
    r.p1 = bits2(__floats2bfloat162_rn(a1, b1));
    r.p2 = bits2(__floats2bfloat162_rn(a1 - __uint_as_float(r.p1 << 16), b1 - __uint_as_float(r.p1 & 0xffff0000u)));
    return r;
}

// Four consecutive k of a row, at most K - 1 of them: beyond the row whatever the last ones are (`f32_within` puts zeros there). No branch stands around a
// load: one behind another's branch it waits for the other. VEC: rows are whole 16-byte words.
template <bool VEC>
__device__ __forceinline__ float4 f32_load(const float* __restrict__ row, int k, int K) {
    float4 v;
    if constexpr (VEC) {
        asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(row + min(k, K - 4)));
    } else {
        v.x = __ldg(row + min(k, K - 1)); v.y = __ldg(row + min(k + 1, K - 1)); v.z = __ldg(row + min(k + 2, K - 1)); v.w = __ldg(row + min(k + 3, K - 1));
    }
    return v;
}
__device__ __forceinline__ void f32_within(float4& v, int k, int K) {
    if (k >= K) v.x = 0.f;
    if (k + 1 >= K) v.y = 0.f;
    if (k + 2 >= K) v.z = 0.f;
    if (k + 3 >= K) v.w = 0.f;
}

// P[3][M][KP] <- the parts of X[M][K], KP = K up to a multiple of 8 (zeros there). Bytes bound it: 10 per element.
template <bool VEC>
__global__ void __launch_bounds__(256) split_rows_kernel(__nv_bfloat16* __restrict__ P, const float* __restrict__ X, int M, int K, int KP) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int words = KP / 8;
    if (i >= (long long)M * words) return;
    const int row = (int)(i / words), k = (int)(i % words) * 8;
    float4 v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {      // written by the kernel before: ordinary loads
        v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* p = X + (size_t)row * K + k + 4 * h;
        if constexpr (VEC) {
            if (k + 4 * h < K) v[h] = *reinterpret_cast<const float4*>(p);
        } else {
            if (k + 4 * h < K) v[h].x = p[0];
            if (k + 4 * h + 1 < K) v[h].y = p[1];
            if (k + 4 * h + 2 < K) v[h].z = p[2];
            if (k + 4 * h + 3 < K) v[h].w = p[3];
        }
    }
    uint32_t o[3][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const Parts a = split2(v[h].x, v[h].y), b = split2(v[h].z, v[h].w);
        o[0][2 * h] = a.p0; o[1][2 * h] = a.p1; o[2][2 * h] = a.p2;
        o[0][2 * h + 1] = b.p0; o[1][2 * h + 1] = b.p1; o[2][2 * h + 1] = b.p2;
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(P + ((size_t)p * M + row) * KP + k) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
}

// Eight columns of both accumulators of a chunk.
__device__ __forceinline__ void f32_tmem_ld(uint32_t at, uint32_t (&r)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t* q = r + 8 * h;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]) : "r"(at + (uint32_t)(h * F32_MAX_TILE)));
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Where parts cannot hold a product (infinities, operands from 2^111 and sums from 2^95 on, which the scale takes out of range) it is made as it is defined: fused multiply-adds in the order of k. A NaN stays one.
__device__ __forceinline__ bool f32_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __noinline__ void f32_again(float* c, const float* __restrict__ a, const float* __restrict__ w, int K) {
    if (f32_finite(*c)) return;
    float s = 0.f;
    for (int k = 0; k < K && s == s; ++k) s = fmaf(a[k], w[k], s);
    *c = s;
}

__device__ __forceinline__ uint32_t f32_in_block(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void f32_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A block per (W tile, tile of bn rows of A) and, where gridDim.z > 1, per segment of k: the segments of a tile are then the blocks of one cluster.
// Warps 0..7 add the accumulators of each chunk to their sums (rows 32 (w % 4).. of W, rows of A in every second sixteen), warps 8..11 split W's even chunks into
// their stage and 12..15 the odd ones, with their next chunk on its way in registers. Warp 16 issues the MMAs, warp 17 fetches A's parts by TMA.
template <bool VEC>
__global__ void __launch_bounds__(F32_THREADS, 1)
gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, const __grid_constant__ CUtensorMap map_a,
                int M, int N, int K, int bn, int slots, int segment, int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* w_stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // swizzle atoms are 1024 B
    unsigned char* a_slots = w_stages + 2 * F32_W_STAGE;
    const int part_bytes = bn * F32_CHUNK * 2, slot_bytes = 3 * part_bytes;
    // Chunk i's two barriers are i % F32_CHUNKS of each: `ready`, when its W is split, its A is here and its accumulators are drained of chunk i - 2; `done`, when its
    // MMAs are: its stage of W and its slot of A are free and its accumulators full. One wait and one commit a chunk: with a barrier for each of these the issuing thread
    // spent 2,800 cycles a chunk, half of them in waits for what was there already, and in three commits (16,384 x 2,048 188 us, 2,048 x 8,192 104).
    uint64_t* ready = reinterpret_cast<uint64_t*>(a_slots + (size_t)slots * slot_bytes);
    uint64_t* done = ready + F32_CHUNKS;
    unsigned char* w_more = reinterpret_cast<unsigned char*>(done + F32_CHUNKS);   // [2][4]: a warp's share of the chunk is not all bf16 numbers
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_more + 8);
    uint32_t* gave_up = tmem_slot + 1;
    static_assert(2 * F32_CHUNKS * 8 + 8 + 8 <= BARRIER_BYTES, "barriers outgrow their space");
    static_assert(F32_MAX_SLOTS <= F32_CHUNKS, "nobody is a whole round of barriers behind");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * 128, m0 = blockIdx.x * bn;
    const bool shared = gridDim.z > 1;
    const int chunks_all = (K + F32_CHUNK - 1) / F32_CHUNK;
    const int begin = shared ? (int)blockIdx.z * segment : 0, end = shared ? min(chunks_all, begin + segment) : chunks_all;

    if (tid == 0) {
        for (int i = 0; i < F32_CHUNKS; ++i) { mbar_init(ready + i, (F32_WORKERS - F32_ADDERS) / 2 + 1 + F32_ADDERS); mbar_init(done + i, 1); }
        *gave_up = 0;
        mbar_fence_init();
    }
    if (warp == F32_WORKERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(4u * F32_MAX_TILE) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    auto is_done = [&](int i) { return mbar_wait(done + i % F32_CHUNKS, (i / F32_CHUNKS) & 1); };
    auto expired = [&](int where) { atomicExch(gave_up, 1u); oxr_report(status, OXR_WAIT_EXPIRED, where); };

    if (warp == F32_WORKERS + 1) {
        // ------------------------------------------------------------------ A's parts
        if (elect_one()) {
            pdl_wait();
            for (int i = 0; i < end - begin; ++i) {
                const int s = i % slots;
                if (i >= slots && !is_done(i - slots)) { expired(60); break; }
                mbar_expect_tx(ready + i % F32_CHUNKS, (uint32_t)slot_bytes);
                for (int p = 0; p < 3; ++p)
                    tma_load_2d(a_slots + (size_t)s * slot_bytes + (size_t)p * part_bytes, &map_a, (begin + i) * F32_CHUNK, p * M + m0, ready + i % F32_CHUNKS);
            }
        }
        __syncwarp();
    } else if (warp == F32_WORKERS) {
        // ------------------------------------------------------------------ MMA
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(128, bn);
            for (int i = 0; i < end - begin; ++i) {
                const int s = i & 1, as = i % slots;
                if (!mbar_wait(ready + i % F32_CHUNKS, (i / F32_CHUNKS) & 1)) { expired(61); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const bool whole = *reinterpret_cast<const volatile uint32_t*>(w_more + 4 * s) != 0;
                const uint32_t w_addr = smem_addr(w_stages + (size_t)s * F32_W_STAGE), a_addr = smem_addr(a_slots + (size_t)as * slot_bytes);
                const uint32_t head = tmem_base + (uint32_t)s * 2 * F32_MAX_TILE, rest = head + F32_MAX_TILE;
                auto product = [&](uint32_t d, int wp, int ap, bool first) {
#pragma unroll
                    for (int k = 0; k < F32_CHUNK / UMMA_K; ++k)
                        umma_bf16(d, umma_desc(w_addr + wp * F32_W_PART + k * UMMA_K * 2), umma_desc(a_addr + ap * part_bytes + k * UMMA_K * 2), idesc, (first && k == 0) ? 0u : 1u);
                };
                product(rest, 0, 2, true);
                if (whole) { product(rest, 2, 0, false); product(rest, 1, 1, false); }
                product(rest, 0, 1, false);
                if (whole) product(rest, 1, 0, false);
                product(head, 0, 0, true);
                umma_commit(done + i % F32_CHUNKS);
            }
        }
        __syncwarp();
    } else if (warp < F32_ADDERS) {
        // ------------------------------------------------------------------ adders
        const int quarter = warp & 3, half = warp >> 2;
        const int col = n0 + quarter * 32 + lane;                    // this lane's row of W: a column of C
        bool ok = true, odd = false;
        if (lane == 0) { mbar_arrive(ready); mbar_arrive(ready + 1); }      // nothing to drain before the first two chunks
        for (int from = 0; from < end - begin && ok; from += segment) {
            const int to = min(end - begin, from + segment);
            float sum[4][16];
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[g][j] = 0.f;
#pragma unroll 1
            for (int i = from; i < to; ++i) {
                const int s = i & 1;
                if (!is_done(i)) { expired(62); ok = false; }
                ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile uint32_t*>(gave_up) == 0);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)s * 2 * F32_MAX_TILE;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const int c0 = (half + 2 * g) * 16;
                    if (c0 < bn) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t v[16];
                            f32_tmem_ld(acc + (uint32_t)(c0 + 8 * h), v);
#pragma unroll
                            for (int j = 0; j < 8; ++j) sum[g][8 * h + j] += __uint_as_float(v[j]) + __uint_as_float(v[8 + j]);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(ready + (i + 2) % F32_CHUNKS);
            }
            if (!ok) break;
            if (shared) {   // every MMA of the block is done: the ring holds the segment's sums now, [bn][128]
                float* mine = reinterpret_cast<float*>(w_stages) + half * 16 * 128 + quarter * 32 + lane;
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    if ((half + 2 * g) * 16 < bn) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) mine[(32 * g + j) * 128] = sum[g][j];
                    }
            } else {        // one block for all segments: each segment's sum is added to what C holds of the ones before it
                pdl_wait();
                const float scale = to == end - begin ? F32_UNSCALE : 1.f;
                int left = col < N ? min(bn, M - m0) - half * 16 : 0;      // rows from this warp's first on
                float* at = C + (size_t)(m0 + half * 16) * N + col;
                asm volatile("" : "+l"(at));   // or the compiler keeps all 64 addresses from segment to segment
#pragma unroll
                for (int g = 0; g < 4; ++g) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j < left) {
                            const float t = (from == 0 ? sum[g][j] : *at + sum[g][j]) * scale;
                            odd = odd || !f32_finite(t);
                            *at = t;
                        }
                        at += N;
                    }
                    at += (size_t)16 * N;
                    left -= 32;
                }
            }
        }
        if (odd) {   // this thread's own stores; the last segment's are what counts
            for (int m = half * 16; m < bn; m = (m & 15) == 15 ? m + 17 : m + 1)
                if (m0 + m < M && col < N) f32_again(C + (size_t)(m0 + m) * N + col, A + (size_t)(m0 + m) * K, W + (size_t)col * K, K);
        }
    } else {
        // ------------------------------------------------------------------ splitters
        const int turn = (warp >> 2) & 1, wrow = (warp & 3) * 2 + (lane >> 4), word = lane & 15;   // rows wrow + 8 p of the tile, k 4 word .. + 3 of a chunk
        bool stale = true;                                           // whether this warp's rows of the stage's second and third parts may not be zero
        float4 v[16];
        unsigned char* stage = w_stages + (size_t)turn * F32_W_STAGE;
        auto fetch = [&](int c) {
            if (c >= end) return;
            if (VEC && (c - begin) % F32_AHEAD == turn && blockIdx.x == 0) {   // the next kilobytes of the rows into L2
                const int k = (c - turn + F32_AHEAD) * F32_CHUNK, bytes = min(F32_AHEAD * F32_CHUNK, min(K, end * F32_CHUNK) - k) * 4;
                const int r = n0 + (warp & 7) * 16 + lane;
                if (lane < 16 && bytes > 0 && r < N) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(W + (size_t)r * K + k), "r"((uint32_t)bytes) : "memory");
            }
#pragma unroll
            for (int p = 0; p < 16; ++p) v[p] = f32_load<VEC>(W + (size_t)min(n0 + wrow + 8 * p, N - 1) * K, c * F32_CHUNK + 4 * word, K);   // rows beyond N: nobody's
        };
        fetch(begin + turn);
        for (int i = turn; begin + i < end; i += 2) {
            bool ok = i < 2 || is_done(i - 2);
            if (!ok) expired(63);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const int k = (begin + i) * F32_CHUNK + 4 * word;
            if ((begin + i + 1) * F32_CHUNK > K) {
#pragma unroll
                for (int p = 0; p < 16; ++p) f32_within(v[p], k, K);
            }
            uint32_t low = 0;
#pragma unroll
            for (int p = 0; p < 16; ++p) low |= __float_as_uint(v[p].x) | __float_as_uint(v[p].y) | __float_as_uint(v[p].z) | __float_as_uint(v[p].w);
            const bool more = __any_sync(0xffffffffu, (low & 0xffffu) != 0);
            unsigned char* at = stage + wrow * 128 + (((word >> 1) ^ wrow) << 4) + (word & 1) * 8;   // rows 8 apart share their swizzle
#pragma unroll
            for (int p = 0; p < 16; ++p, at += 8 * 128) {
                if (more) {
                    const Parts a = split2(v[p].x, v[p].y), b = split2(v[p].z, v[p].w);
                    *reinterpret_cast<uint2*>(at) = make_uint2(a.p0, b.p0);
                    *reinterpret_cast<uint2*>(at + F32_W_PART) = make_uint2(a.p1, b.p1);
                    *reinterpret_cast<uint2*>(at + 2 * F32_W_PART) = make_uint2(a.p2, b.p2);
                } else {
                    *reinterpret_cast<uint2*>(at) = make_uint2(__byte_perm(__float_as_uint(F32_SCALE * v[p].x), __float_as_uint(F32_SCALE * v[p].y), 0x7632),
                                                               __byte_perm(__float_as_uint(F32_SCALE * v[p].z), __float_as_uint(F32_SCALE * v[p].w), 0x7632));
                    if (stale) {
                        *reinterpret_cast<uint2*>(at + F32_W_PART) = make_uint2(0, 0);
                        *reinterpret_cast<uint2*>(at + 2 * F32_W_PART) = make_uint2(0, 0);
                    }
                }
            }
            stale = more;
            if (lane == 0) w_more[4 * turn + (warp & 3)] = more;
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + i % F32_CHUNKS);
            fetch(begin + i + 2);   // behind the fence, which would wait for loads on their way
        }
    }
    if (shared) {
        f32_cluster_sync();
        pdl_wait();
        // block z adds the segments' sums of its share of the rows, in order
        const uint32_t mine = smem_addr(w_stages);
        const int ranks = gridDim.z, rank = blockIdx.z;
        for (int e = rank * F32_THREADS + tid; e < bn * 128; e += ranks * F32_THREADS) {
            const int m = m0 + e / 128, n = n0 + e % 128;
            if (m >= M || n >= N) continue;
            float t = 0.f;
            for (int r = 0; r < ranks; ++r) {
                float v;
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(f32_in_block(mine, (uint32_t)r) + 4u * (uint32_t)e));
                t = r == 0 ? v : t + v;
            }
            t *= F32_UNSCALE;
            C[(size_t)m * N + n] = t;
            if (!f32_finite(t)) f32_again(C + (size_t)m * N + n, A + (size_t)m * K, W + (size_t)n * K, K);
        }
        f32_cluster_sync();   // no block leaves while another may still read its shared memory
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == F32_WORKERS) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(4u * F32_MAX_TILE) : "memory");
    }
}

// Segments of k that have a sum of their own: by K alone, so that an element's result depends on nothing else.
int f32_segments(int K) {
    const int n = K / F32_MIN_SEGMENT;
    return n < 1 ? 1 : n > F32_MAX_SEGMENTS ? F32_MAX_SEGMENTS : n;
}

template <bool VEC>
int launch_f32(float* C, const float* A, const float* W, __nv_bfloat16* parts, int M, int N, int K, int tile, bool shared, int* status, cudaStream_t stream) {
    static int attr = -1;   // per instantiation
    if (attr != 0) {
        attr = (int)cudaFuncSetAttribute(gemm_f32_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (attr != 0) return 1000 + attr;
    }
    const int KP = (K + 7) / 8 * 8;
    CUtensorMap map;
    if (!oxr_make_map_bf16(&map, parts, 3ull * M, KP, tile)) return OXR_BAD_ARGUMENT;
    const long long words = (long long)M * (KP / 8);
    const dim3 split_grid((unsigned)((words + 255) / 256));
    if (K % 4 == 0 && (uintptr_t)A % 16 == 0) oxr_launch_small(split_rows_kernel<true>, split_grid, dim3(256), 0, stream, parts, A, M, K, KP);
    else oxr_launch_small(split_rows_kernel<false>, split_grid, dim3(256), 0, stream, parts, A, M, K, KP);
    const int code = oxr_launch_status();
    if (code != 0) return code;

    const int chunks = (K + F32_CHUNK - 1) / F32_CHUNK, want = f32_segments(K);
    const int segment = (chunks + want - 1) / want, segments = (chunks + segment - 1) / segment;
    int slots = (RING_BYTES - 2 * F32_W_STAGE) / (3 * tile * F32_CHUNK * 2);
    if (slots > F32_MAX_SLOTS) slots = F32_MAX_SLOTS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((M + tile - 1) / tile, (N + 127) / 128, shared ? segments : 1);
    if (cfg.gridDim.y > 65535) return OXR_BAD_ARGUMENT;
    cfg.blockDim = dim3(F32_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    int n = 0;
    if (shared && segments > 1) {
        attrs[n].id = cudaLaunchAttributeClusterDimension;
        attrs[n].val.clusterDim.x = 1;
        attrs[n].val.clusterDim.y = 1;
        attrs[n].val.clusterDim.z = (unsigned)segments;
        ++n;
    }
    if (oxr_chain_kernels) {
        attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attrs;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, gemm_f32_kernel<VEC>, C, A, W, map, M, N, K, tile, slots, segment, status);
    return oxr_launch_status();
}
}  // namespace

// gemm_f32_short.cu
OXR_API int oxr_gemm_f32_is_short(int N, int K);
int oxr_gemm_f32_short(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream);

// Short products (`oxr_gemm_f32_is_short`) run a kernel of their own, which uses none of the arguments after K. parts: 3 * M * (K up to a multiple of 8) bf16 numbers of scratch, 16-byte aligned. tile: rows of A per block, a multiple of 16 from 16 to 128. shared: the
// segments of k go to the blocks of a cluster; the results are the same.
OXR_API int oxr_gemm_f32_nt(float* C, const float* A, const float* W, void* parts, int M, int N, int K, int tile, int shared, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K > 0 && oxr_gemm_f32_is_short(N, K)) return oxr_gemm_f32_short(C, A, W, M, N, K, stream);
    if (K <= 0 || tile < 16 || tile > F32_MAX_TILE || tile % 16 != 0 || (uintptr_t)parts % 16 != 0) return OXR_BAD_ARGUMENT;
    if (3ll * M > 0x7fffffffll) return OXR_BAD_ARGUMENT;
    if (K % 4 == 0 && (uintptr_t)W % 16 == 0) return launch_f32<true>(C, A, W, (__nv_bfloat16*)parts, M, N, K, tile, shared != 0, status, stream);
    return launch_f32<false>(C, A, W, (__nv_bfloat16*)parts, M, N, K, tile, shared != 0, status, stream);
}

OXR_API int oxr_gemm_f32_segments(int K) { return f32_segments(K); }

// How many clusters of `segments` blocks of the product the GPU holds at a time (0 if such a cluster cannot be launched).
OXR_API int oxr_gemm_f32_max_clusters(int segments) {
    if (segments < 1 || segments > F32_MAX_SEGMENTS) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 64, (unsigned)segments);
    cfg.blockDim = dim3(F32_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = (unsigned)segments;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(gemm_f32_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_f32_kernel<true>, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}
