// Gated linear attention between its in- and out-projections: a recurrence whose state decays per key channel.
//
// Per request and head the state is a matrix S [DK, DV] (zero for a new request; one fp32 row per request holds S of every head). With
// a decay per key channel alpha_t = sigmoid(z_t)^(1 / tau), z_t = (the decay projection) + bias:
//
//   S_t = diag(alpha_t) S_(t-1) + k_t v_t^T          o_t = S_t^T q_t          q_t already scaled
//
// The decay (log-sigmoid, division by tau, exponential), S and every sum over it are fp32; T is the activation type of the q|k|v
// projections; z is fp32. The recurrence runs token by token in the order of the sequence whatever the cut, and every kernel for it (the ones
// below, and the one of scan_columns.cuh) adds up o in one order, so a position's result does not depend on how a prompt was cut into steps nor on
// what else is in the batch. Columns of S (one value dimension each) are independent: a block takes 32 columns of one head of one request.
//
// grid (ceil(DV / 32), heads, requests); block = 32 * NW threads with NW = ceil(DK / KPT). Lane l owns the value column p = 32 blockIdx.x + l,
// warp w the key entries 4 (w + NW m) .. + 3 for m = 0 .. KPT / 4 - 1: a thread keeps KPT = 32 or 16 entries of S in registers (16: twice the warps for the same
// state, which is what hides the loop's latencies when a step brings many tokens of a request; keys of up to 128). A tile of TT tokens goes through shared memory at
// a time (thread d brings entry d of k, q and the decay of each token; the next tile's loads are in flight while this one is computed); the
// warps' partial sums of S^T q meet in shared memory and are added after the tile. Every NW-th four entries to a warp, so that a thread's sums are the
// first ones of the order in scan_columns.cuh.
#include <climits>

#include "scan_columns.cuh"

__device__ __forceinline__ float gla_log_sigmoid(float v) { return fminf(v, 0.f) - log1pf(expf(-fabsf(v))); }

// The bound on registers: twelve warps an SM (16 with eight warps of 16 entries), without it the compiler takes registers for eight. Single tokens of 48
// requests, 16 heads of 128 x 256: 59 us, 80 without the bound.
template <typename T, int NW, int TT, int KPT>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? (KPT == 32 ? 1 : 2) : 12 / NW) gla_scan_kernel(
    float* __restrict__ y, const T* __restrict__ proj, int proj_stride, int q_col0, int k_col0, int v_col0, const float* __restrict__ z,
    const float* __restrict__ z_bias, float inv_tau, int heads, int DK, int DV, float q_scale, float* __restrict__ state, long long slot_stride,
    const int* __restrict__ cu_q, const int* __restrict__ state_slots, int most) {
    constexpr int DKP = KPT * NW, NT = 32 * NW;      // NT >= DKP: thread d brings key entry d of every token
    __shared__ __align__(16) float ks[TT][DKP];
    __shared__ __align__(16) float qs[TT][DKP];
    __shared__ __align__(16) float as[TT][DKP];
    __shared__ float vs[TT][32], part[TT][NW][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = threadIdx.x;
    const int p0 = blockIdx.x * 32, p = p0 + lane, h = blockIdx.y, r = blockIdx.z;
    const int t0 = cu_q[r], t1 = cu_q[r + 1];
    if (t1 <= t0 || t1 - t0 > most) return;          // requests of more tokens are the other kernel's of this step
    float* S = state + (long long)state_slots[r] * slot_stride + (long long)h * DK * DV;
    f32x2 s[KPT / 2];                                // pair i: entries entry(i) and entry(i) + 1
    auto entry = [&](int i) { return 4 * (warp + NW * (i >> 1)) + 2 * (i & 1); };
    auto stored = [&](int e) { return (e < DK && p < DV) ? S[(size_t)e * DV + p] : 0.f; };
#pragma unroll
    for (int i = 0; i < KPT / 2; ++i) s[i] = pack2(stored(entry(i)), stored(entry(i) + 1));
    const float zb = n < DK ? z_bias[h * DK + n] : 0.f;

    constexpr int VPT = (TT * 32 + NT - 1) / NT;      // v values per thread and tile
    T kreg[TT], qreg[TT], vreg[VPT];
    float zreg[TT];
    auto fetch = [&](int tile) {
        const int nt = min(TT, t1 - tile);
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            const bool ok = t < nt && n < DK;
            const size_t tok = (size_t)(tile + (t < nt ? t : 0));
            const T* row = proj + tok * proj_stride;
            kreg[t] = ok ? row[k_col0 + h * DK + n] : Num<T>::from_f32(0.f);
            qreg[t] = ok ? row[q_col0 + h * DK + n] : Num<T>::from_f32(0.f);
            zreg[t] = ok ? z[tok * heads * DK + h * DK + n] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int i = n + j * NT, t = i >> 5, c = i & 31;
            vreg[j] = (t < nt && p0 + c < DV) ? proj[(size_t)(tile + t) * proj_stride + v_col0 + h * DV + p0 + c] : Num<T>::from_f32(0.f);
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            if (n < DKP) {
                ks[t][n] = Num<T>::to_f32(kreg[t]);
                qs[t][n] = Num<T>::to_f32(qreg[t]);
                as[t][n] = expf(gla_log_sigmoid(zreg[t] + zb) * inv_tau);
            }
        }
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int i = n + j * NT;
            if (i < TT * 32) vs[i >> 5][i & 31] = Num<T>::to_f32(vreg[j]);
        }
    };
    fetch(t0);
    stash();
    __syncthreads();
    for (int tile = t0; tile < t1; tile += TT) {
        const int nt = min(TT, t1 - tile);
        const bool more = tile + TT < t1;
        if (more) fetch(tile + TT);
        for (int t = 0; t < nt; ++t) {
            const float tv = vs[t][lane];
            const f32x2 tv2 = pack2(tv, tv);
            float four[KPT / 4];
#pragma unroll
            for (int m = 0; m < KPT / 4; ++m) {
                const int e = entry(2 * m);
                const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(&ks[t][e]), qq = *reinterpret_cast<const ulonglong2*>(&qs[t][e]),
                                 aa = *reinterpret_cast<const ulonglong2*>(&as[t][e]);
                s[2 * m] = fma2(aa.x, s[2 * m], mul2(kk.x, tv2));
                s[2 * m + 1] = fma2(aa.y, s[2 * m + 1], mul2(kk.y, tv2));
                four[m] = scan_sum_four(s[2 * m], s[2 * m + 1], qq.x, qq.y);
            }
            part[t][warp][lane] = scan_halve<KPT / 4>(four);
        }
        __syncthreads();
        for (int i = n; i < nt * 32; i += NT) {
            const int t = i >> 5, c = i & 31;
            if (p0 + c < DV) {
                float v[NW];
#pragma unroll
                for (int w = 0; w < NW; ++w) v[w] = part[t][w][c];
                y[(size_t)(tile + t) * heads * DV + h * DV + p0 + c] = scan_halve<NW>(v) * q_scale;
            }
        }
        if (more) {
            __syncthreads();   // the tile's sums have been read
            stash();
            __syncthreads();
        }
    }
    if (p < DV) {
#pragma unroll
        for (int i = 0; i < KPT / 2; ++i) {
            float lo, hi;
            unpack2(s[i], lo, hi);
            if (entry(i) < DK) S[(size_t)entry(i) * DV + p] = lo;
            if (entry(i) + 1 < DK) S[(size_t)(entry(i) + 1) * DV + p] = hi;
        }
    }
}

// decay[t, i] = sigmoid(z[t, i] + bias[i])^(1 / tau), four entries a thread: once per token and key channel, where the recurrence's blocks (one per 32 value
// columns) would each work it out again
__global__ void gla_decay_kernel(float4* __restrict__ decay, const float4* __restrict__ z, const float4* __restrict__ z_bias, float inv_tau, int width4, size_t total) {
    pdl_wait();
    pdl_trigger();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const float4 v = z[i], b = z_bias[i % width4];
    decay[i] = make_float4(expf(gla_log_sigmoid(v.x + b.x) * inv_tau), expf(gla_log_sigmoid(v.y + b.y) * inv_tau), expf(gla_log_sigmoid(v.z + b.z) * inv_tau),
                           expf(gla_log_sigmoid(v.w + b.w) * inv_tau));
}

// n_long requests bring at least long_from tokens; long_list (host memory, may be null) names them, the longest first. With `decay` (fp32 scratch
// [n_tokens, heads * DK]) they go to the kernel of scan_columns.cuh, where that takes the sizes, all others to the kernel above, in a launch of its own.
// Which kernel takes a request changes no result.
OXR_API int oxr_gla_scan(float* y, const void* proj, int n_requests, int proj_stride, int q_col0, int k_col0, int v_col0, const float* z,
                         const float* z_bias, float tau, int heads, int DK, int DV, float q_scale, float* state, long long slot_stride, const int* cu_q,
                         const int* state_slots, int dtype, int key_entries_per_thread, float* decay, int n_tokens,
                         const int* long_list, int n_long, int long_from, cudaStream_t stream) {
    if (n_requests <= 0) return 0;
    if (heads <= 0 || DK <= 0 || DK > 256 || DV <= 0 || heads > 65535 || n_requests > 65535 || !(tau > 0.f)) return OXR_BAD_ARGUMENT;
    int most = INT_MAX;
    if (decay != nullptr && n_tokens > 0 && n_long > 0) {
        const size_t size = dtype == 0 ? 4 : 2;
        ScanArgs a = {};
        a.k = (const char*)proj + k_col0 * size; a.q = (const char*)proj + q_col0 * size; a.x = (const char*)proj + v_col0 * size;
        a.stride = proj_stride; a.k_group = 1; a.decay = decay; a.q_scale = q_scale; a.y = y; a.state = state; a.slot_stride = slot_stride; a.cu_q = cu_q;
        a.state_slots = state_slots; a.heads = heads; a.DV = DV; a.n_requests = n_requests;
        a.least = n_long < n_requests ? long_from : 0;
        a.order = RequestOrder(long_list, n_long);
        if ((dtype == 0 ? scan_fits<float>(a, DK) : scan_fits<__nv_bfloat16>(a, DK)) && (uintptr_t)z % 16 == 0 && (uintptr_t)z_bias % 16 == 0) {
            const size_t total = (size_t)n_tokens * heads * DK / 4;
            oxr_launch_small(gla_decay_kernel, dim3((unsigned)((total + 127) / 128)), dim3(128), 0, stream, (float4*)decay, (const float4*)z, (const float4*)z_bias, 1.f / tau,
                                                                                 heads * DK / 4, total);
            int rc = oxr_launch_status();
            if (rc) return rc;
            rc = dtype == 0 ? scan_launch<float, true>(a, DK, n_long, stream) : scan_launch<__nv_bfloat16, true>(a, DK, n_long, stream);
            if (rc || n_long >= n_requests) return rc;
            most = long_from - 1;
        }
    }
    dim3 grid((DV + 31) / 32, heads, n_requests);
    // key_entries_per_thread 16 or 32 forces a split. Else 16 (twice the warps per head) for portions of prompts, where that still fits a block of 8 warps; for few
    // tokens the state's trip through the registers is all there is, and fewer partial sums are cheaper (8 single tokens: 20.5 against 24.6 us)
    const bool narrow = DK <= 128 && (key_entries_per_thread ? key_entries_per_thread == 16 : n_long > 0 && most == INT_MAX);
    const int nw = narrow ? (DK + 15) / 16 : (DK + 31) / 32;
#define OXR_GLA(T, NW) \
    do { \
        if (narrow) oxr_launch(gla_scan_kernel<T, NW, 8, 16>, dim3(grid), dim3(32 * NW), 0, stream, false, y, (const T*)proj, proj_stride, q_col0, k_col0, v_col0, z, z_bias, 1.f / tau, \
                                                                                heads, DK, DV, q_scale, state, slot_stride, cu_q, state_slots, most); \
        else oxr_launch(gla_scan_kernel<T, NW, 8, 32>, dim3(grid), dim3(32 * NW), 0, stream, false, y, (const T*)proj, proj_stride, q_col0, k_col0, v_col0, z, z_bias, 1.f / tau, heads, \
                                                                         DK, DV, q_scale, state, slot_stride, cu_q, state_slots, most); \
    } while (0)
#define OXR_GLA_T(T) \
    do { \
        if (nw <= 1) OXR_GLA(T, 1); \
        else if (nw <= 2) OXR_GLA(T, 2); \
        else if (nw <= 4) OXR_GLA(T, 4); \
        else OXR_GLA(T, 8); \
    } while (0)
    if (dtype == 0) OXR_GLA_T(float);
    else OXR_GLA_T(__nv_bfloat16);
#undef OXR_GLA_T
#undef OXR_GLA
    return oxr_launch_status();
}
