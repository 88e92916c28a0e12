// True fp32 GEMM on the CUDA cores: C[M,N] = A[M,K] * W[N,K]^T, fp32 FMA accumulation, no TF32.
//
// This is the matrix product of the 32-bit path of the whole model (the reference multiplies through
// nn.Linear, oxr_runtime/language.py:223-244; in fp32 only on the CPU in its tests). Every output element is
// the sum over k = 0, 1, 2, ... of a[m,k] * w[n,k] accumulated in that order with fused multiply-adds,
// whatever the tile shape and whatever else is in the batch: a row's result does not depend on M.
#include "common.cuh"

// At most 16 rows: 16 x 64 tiles, four columns of one row per thread (few blocks of little work; latency, not the FMA rate, bounds it).
__global__ void __launch_bounds__(256) gemm_f32_few_kernel(float* __restrict__ C, const float* __restrict__ A,
                                                           const float* __restrict__ W, int M, int N, int K) {
    constexpr int BM = 16, BN = 64, BK = 16, TM = BM / 16, TN = 4;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int i = tid; i < BM * BK; i += 256) {
            const int r = i / BK, k = i % BK;
            const int gm = m0 + r, gk = k0 + k;
            As[k][r] = (gm < M && gk < K) ? A[(size_t)gm * K + gk] : 0.f;
        }
        for (int i = tid; i < BN * BK; i += 256) {
            const int r = i / BK, k = i % BK;
            const int gn = n0 + r, gk = k0 + k;
            Ws[k][r] = (gn < N && gk < K) ? W[(size_t)gn * K + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn < N) C[(size_t)gm * N + gn] = acc[i][j];
        }
    }
}

// More rows: tiles of 8 TM x 16 TN on 128 threads, TM x TN sums per thread. What bounds it is the FMA rate (128 lanes of an SM,
// 74 TFLOP/s at the full clock), so everything else has to stay out of the way of the multiply-adds:
//  * sums in pairs of columns with fma.rn.f32x2 (each half rounds as fmaf does): half the issue slots, which leaves room for the loads and for doubling
//    a[m] in registers (kept twice in shared memory, as it was first, its loads took longer than the multiply-adds);
//  * a thread's columns lie V apart in groups (group j of a thread starts at V (16 j + tx)), so that a warp reads consecutive words;
//  * the next 16 k of A and W are fetched into registers while the current ones are multiplied, and put into the other half of a
//    double buffer: one barrier per 16 k.
// Four warps fill an SM's four schedulers by themselves. The tile is chosen by the launcher, see there.
// 333 rows on a B200, against 64 x 64 tiles of 4 x 4 a thread filled element by element: 3,072 x 2,048 127 us (324), 2,048 x 2,048 109 (315),
// 16,384 x 2,048 530 (1,403), 2,048 x 8,192 433 (1,477): 26 to 42 TFLOP/s. Stages of 32 k instead of 16 cost registers and with them blocks: slower.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

constexpr int F32_BK = 16, F32_THREADS = 128;

// VEC: rows of A and W are whole 16-byte words (K a multiple of 4, aligned bases).
template <int TM, int TN, bool VEC>
__global__ void __launch_bounds__(F32_THREADS) gemm_f32_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                                                                    int M, int N, int K) {
    constexpr int BK = F32_BK, BM = 8 * TM, BN = 16 * TN;
    constexpr int V = TN % 4 == 0 ? 4 : 2, G = TN / V, RV = TM % 4 == 0 ? 4 : 2;                     // columns per group, groups per thread
    constexpr int LA = BM + 4, LW = BN + 4;                            // floats per k of the two tiles
    constexpr int QA = (BM * 4 + F32_THREADS - 1) / F32_THREADS, QW = (BN * 4 + F32_THREADS - 1) / F32_THREADS;   // 16-byte words per thread
    static_assert(TM % 2 == 0 && TN % 2 == 0, "rows and columns come in pairs");
    __shared__ __align__(16) float As[2][BK * LA];
    __shared__ __align__(16) float Ws[2][BK * LW];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float4 ra[QA], rw[QW];
    // four consecutive k of one row; zeros beyond the matrix
    auto fetch = [&](const float* __restrict__ X, int row, int rows, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= rows || k >= K) return v;
        const float* p = X + (size_t)row * K + k;
        if constexpr (VEC) return __ldg(reinterpret_cast<const float4*>(p));
        v.x = p[0];
        if (k + 1 < K) v.y = p[1];
        if (k + 2 < K) v.z = p[2];
        if (k + 3 < K) v.w = p[3];
        return v;
    };
    auto fetch_tiles = [&](int k0) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int q = tid + i * F32_THREADS;
            if (q < BM * 4) ra[i] = fetch(A, m0 + (q >> 2), M, k0 + (q & 3) * 4);
        }
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const int q = tid + i * F32_THREADS;
            if (q < BN * 4) rw[i] = fetch(W, n0 + (q >> 2), N, k0 + (q & 3) * 4);
        }
    };
    auto put_tiles = [&](int b) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int q = tid + i * F32_THREADS;
            if (q >= BM * 4) break;
            const float e[4] = {ra[i].x, ra[i].y, ra[i].z, ra[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) As[b][((q & 3) * 4 + j) * LA + (q >> 2)] = e[j];
        }
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const int q = tid + i * F32_THREADS;
            if (q >= BN * 4) break;
            const float e[4] = {rw[i].x, rw[i].y, rw[i].z, rw[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) Ws[b][((q & 3) * 4 + j) * LW + (q >> 2)] = e[j];
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    fetch_tiles(0);
    put_tiles(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK) {
        const bool more = k0 + BK < K;
        if (more) fetch_tiles(k0 + BK);
        const float* as = As[buf] + TM * ty;
        const float* ws = Ws[buf] + V * tx;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            unsigned long long a[TM], b[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += RV) {      // one word feeds RV rows; each is doubled in registers
                if constexpr (RV == 4) {
                    const float4 p = *reinterpret_cast<const float4*>(as + k * LA + i);
                    a[i] = pack2(p.x, p.x); a[i + 1] = pack2(p.y, p.y); a[i + 2] = pack2(p.z, p.z); a[i + 3] = pack2(p.w, p.w);
                } else {
                    const float2 p = *reinterpret_cast<const float2*>(as + k * LA + i);
                    a[i] = pack2(p.x, p.x); a[i + 1] = pack2(p.y, p.y);
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if constexpr (V == 4) {
                    const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(ws + k * LW + 64 * g);
                    b[2 * g] = p.x;
                    b[2 * g + 1] = p.y;
                } else {
                    b[g] = *reinterpret_cast<const unsigned long long*>(ws + k * LW + 32 * g);
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], a[i], b[j]);
        }
        buf ^= 1;
        if (more) put_tiles(buf);   // the half that every thread left before the last barrier
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            const int gn = n0 + (j * 2 / V) * 16 * V + V * tx + j * 2 % V;
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][j]));
            if (gn < N) C[(size_t)gm * N + gn] = lo;
            if (gn + 1 < N) C[(size_t)gm * N + gn + 1] = hi;
        }
    }
}

template <int TM, int TN>
int launch_f32(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    dim3 grid((N + 16 * TN - 1) / (16 * TN), (M + 8 * TM - 1) / (8 * TM));
    if (grid.y > 65535) return OXR_BAD_ARGUMENT;
    if (K % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) gemm_f32_tile_kernel<TM, TN, true><<<grid, F32_THREADS, 0, stream>>>(C, A, W, M, N, K);
    else gemm_f32_tile_kernel<TM, TN, false><<<grid, F32_THREADS, 0, stream>>>(C, A, W, M, N, K);
    return oxr_launch_status();
}

// Tile shapes (TM, TN) and what a k costs, in tenths of a nanosecond, measured on a B200: `loaded`, a tile's share of an SM that is full of them (1,000 rows
// x 16,384 columns); `lone`, a tile alone on its SM, which waits for its own loads and barriers (40 rows x 2,048 columns). Between the two
// n tiles on an SM take n * loaded + (lone - loaded) / n: within 8 % of what 40 to 1,000 rows by 2,048 to 32,768 columns measured, for every shape.
struct F32Tile { int tm, tn; float loaded, lone; };
constexpr F32Tile F32_TILES[] = {{8, 8, 465, 595}, {8, 6, 365, 520}, {6, 8, 390, 545}, {6, 6, 307, 440}, {8, 4, 271, 460}, {6, 4, 231, 450}, {4, 4, 190, 480}, {2, 4, 159, 340}};

OXR_API int oxr_gemm_f32_nt(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return OXR_BAD_ARGUMENT;
    if (M <= 16) {
        gemm_f32_few_kernel<<<dim3((N + 63) / 64), 256, 0, stream>>>(C, A, W, M, N, K);
        return oxr_launch_status();
    }
    // The SM that gets the most tiles decides. A few hundred rows make few large tiles (2,048 columns: 96 of 64 x 128 on 148 SMs), smaller ones fill
    // the chip better: 100 rows x 2,048 columns, k 8,192: 297 us in tiles of 16 x 64, 425 in tiles of 32 x 64, 489 in tiles of 64 x 128.
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    int best = 0;
    float best_cost = -1.f;
    for (int i = 0; i < (int)(sizeof(F32_TILES) / sizeof(F32_TILES[0])); ++i) {
        const F32Tile& t = F32_TILES[i];
        const long long tiles = (long long)((M + 8 * t.tm - 1) / (8 * t.tm)) * ((N + 16 * t.tn - 1) / (16 * t.tn));
        const float n = (float)((tiles + sms - 1) / sms), cost = n * t.loaded + (t.lone - t.loaded) / n;
        if (best_cost < 0.f || cost < best_cost) { best = i; best_cost = cost; }
    }
    switch (best) {
        case 0: return launch_f32<8, 8>(C, A, W, M, N, K, stream);
        case 1: return launch_f32<8, 6>(C, A, W, M, N, K, stream);
        case 2: return launch_f32<6, 8>(C, A, W, M, N, K, stream);
        case 3: return launch_f32<6, 6>(C, A, W, M, N, K, stream);
        case 4: return launch_f32<8, 4>(C, A, W, M, N, K, stream);
        case 5: return launch_f32<6, 4>(C, A, W, M, N, K, stream);
        case 6: return launch_f32<4, 4>(C, A, W, M, N, K, stream);
        default: return launch_f32<2, 4>(C, A, W, M, N, K, stream);
    }
}
