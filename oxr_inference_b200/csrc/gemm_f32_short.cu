// 32-bit products of short rows and small weights: C[M,N] = A[M,K] * W[N,K]^T, every element summed in 64 bits and rounded once.
//
// The tensor-core product of gemm_f32.cu splits its rows in a launch of its own and sets up barriers and tensor memory before the first multiply: 7.5 us at least. Here a
// block stages 16 or 32 k of its rows of A and W at a time as doubles (a product of two fp32 numbers is exact in one), and a thread keeps TM x TN sums, the even and the odd k
// apart. That is one order, whatever the tile, so a row's result does not depend on M; the error is one rounding to 32 bits.
// What bounds it: a stage's trip to memory and its two barriers, 0.9 us, while there is less than a round of blocks; 64-bit multiply-adds beyond (18 TFLOP/s). 333 rows, in a
// graph, us, gemm_f32.cu, here and tiles of 32-bit multiply-adds: 64 x 64 8.0, 3.4, 3.5; 16 x 256 12.2, 9.4, 7.8; 2,048 x 16 9.0, 5.1, 3.1; one row of 64 x 64 8.0, 3.3, 7.0.
#include "common.cuh"

namespace {
// A block of 16 x 16 threads: tile 16 TM rows x 16 TN columns. A thread has the rows TM ty .. and, in pairs 32 apart, the columns 2 tx, 2 tx + 1 (TN 2, 4).
template <int TM, int TN, int SH_BK, bool VEC>
__global__ void __launch_bounds__(256) gemm_f32_short_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K) {
    pdl_wait();
    pdl_trigger();
    constexpr int BM = 16 * TM, BN = 16 * TN, LA = BM + 2, LW = BN + 2;      // doubles per k; even, for loads of two
    constexpr int QA = (BM * (SH_BK / 4) + 255) / 256, QW = (BN * (SH_BK / 4) + 255) / 256;   // words of four k per thread
    static_assert(TN % 2 == 0, "columns come in pairs");
    __shared__ __align__(16) double As[SH_BK * LA], Ws[SH_BK * LW];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float4 ra[QA], rw[QW];
    // four consecutive k of a row, zeros beyond the matrix
    auto fetch = [&](const float* __restrict__ X, int row, int rows, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= rows || k >= K) return v;
        const float* p = X + (size_t)row * K + k;
        if constexpr (VEC) return *reinterpret_cast<const float4*>(p);
        v.x = p[0];
        if (k + 1 < K) v.y = p[1];
        if (k + 2 < K) v.z = p[2];
        if (k + 3 < K) v.w = p[3];
        return v;
    };
    auto fetch_stage = [&](int k0) {
#pragma unroll
        for (int i = 0; i < QA; ++i) {
            const int q = tid + 256 * i;
            if (q < BM * (SH_BK / 4)) ra[i] = fetch(A, m0 + q / (SH_BK / 4), M, k0 + q % (SH_BK / 4) * 4);
        }
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const int q = tid + 256 * i;
            if (q < BN * (SH_BK / 4)) rw[i] = fetch(W, n0 + q / (SH_BK / 4), N, k0 + q % (SH_BK / 4) * 4);
        }
    };
    auto put = [&](double* dst, int ld, int q, const float4& v) {
        double* at = dst + (size_t)(q % (SH_BK / 4)) * 4 * ld + q / (SH_BK / 4);
        at[0] = (double)v.x; at[ld] = (double)v.y; at[2 * ld] = (double)v.z; at[3 * ld] = (double)v.w;
    };

    double acc[2][TM][TN];      // even and odd k: one sum's multiply-adds wait for one another
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[1][i][j] = 0.0;
    fetch_stage(0);
    for (int k0 = 0; k0 < K; k0 += SH_BK) {
        if (k0 > 0) __syncthreads();   // the stage before is read
#pragma unroll
        for (int i = 0; i < QA; ++i)
            if (tid + 256 * i < BM * (SH_BK / 4)) put(As, LA, tid + 256 * i, ra[i]);
#pragma unroll
        for (int i = 0; i < QW; ++i)
            if (tid + 256 * i < BN * (SH_BK / 4)) put(Ws, LW, tid + 256 * i, rw[i]);
        __syncthreads();
        if (k0 + SH_BK < K) fetch_stage(k0 + SH_BK);
        const int depth = min(SH_BK, K - k0);
#pragma unroll 4
        for (int k = 0; k < depth; k += 2) {      // an odd K ends in a k of zeros
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double a[TM];
                double2 b[TN / 2];
                if constexpr (TM % 2 == 0) {
#pragma unroll
                    for (int i = 0; i < TM; i += 2) {
                        const double2 p = *reinterpret_cast<const double2*>(As + (k + h) * LA + TM * ty + i);
                        a[i] = p.x;
                        a[i + 1] = p.y;
                    }
                } else {
                    a[0] = As[(k + h) * LA + ty];
                }
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) b[j] = *reinterpret_cast<const double2*>(Ws + (k + h) * LW + 2 * tx + 32 * j);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) {
                        acc[h][i][2 * j] = fma(a[i], b[j].x, acc[h][i][2 * j]);
                        acc[h][i][2 * j + 1] = fma(a[i], b[j].y, acc[h][i][2 * j + 1]);
                    }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + TM * ty + i;
        if (m >= M) break;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + 2 * tx + 32 * (j / 2) + j % 2;
            if (n < N) C[(size_t)m * N + n] = (float)(acc[0][i][j] + acc[1][i][j]);
        }
    }
}

template <int TM, int TN, int SH_BK>
int launch_short(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + 16 * TN - 1) / (16 * TN), (M + 16 * TM - 1) / (16 * TM));
    if (grid.y > 65535) return OXR_BAD_ARGUMENT;
    if (K % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) oxr_launch_small(gemm_f32_short_kernel<TM, TN, SH_BK, true>, grid, dim3(256), 0, stream, C, A, W, M, N, K);
    else oxr_launch_small(gemm_f32_short_kernel<TM, TN, SH_BK, false>, grid, dim3(256), 0, stream, C, A, W, M, N, K);
    return oxr_launch_status();
}
}  // namespace

// Whether a product goes this way: by the weight's shape alone, so that a row's result does not depend on M. The line lies where this kernel is the faster one for every M
// from 1 to 8,192: beyond it, it still is for few rows (17 of 2,048 x 64 3.4 us, gemm_f32.cu 8.3) and no longer for many (2,048 rows: 37 and 19).
OXR_API int oxr_gemm_f32_is_short(int N, int K) { return K <= 16 || (K <= 256 && (long long)N * K <= 4096); }

int oxr_gemm_f32_short(float* C, const float* A, const float* W, int M, int N, int K, cudaStream_t stream) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    // the largest tile of which there is one for every SM
    if ((long long)((M + 127) / 128) * ((N + 63) / 64) >= sms) return launch_short<8, 4, 16>(C, A, W, M, N, K, stream);
    if ((long long)((M + 63) / 64) * ((N + 63) / 64) >= sms) return launch_short<4, 4, 32>(C, A, W, M, N, K, stream);
    if ((long long)((M + 31) / 32) * ((N + 31) / 32) >= sms) return launch_short<2, 2, 32>(C, A, W, M, N, K, stream);
    return launch_short<1, 2, 32>(C, A, W, M, N, K, stream);
}
