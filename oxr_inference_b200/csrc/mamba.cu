// A Mamba-2 (state-space duality) mixer's kernels between its in- and out-projection: the short causal convolution
// with SiLU, the roll of the convolution's tail, the selective-state recurrence, and the gated grouped RMSNorm.
//
// A step brings, per request, any number of new tokens (a portion of a prompt, or one decoded token); what earlier steps
// left is the per-request state in a slot: the recurrence's S [heads, N, vdim] and the last taps-1 inputs of the
// convolution [channels, taps-1], both fp32. Everything that enters the recurrence is fp32: dt = softplus(dt + bias)
// (no clamp), the decay exp(-exp(A_log) dt), S itself and the sums over it. T is the activation type of the projections.
//
//   S_t = decay_t S_(t-1) + dt_t B_t x_t^T          y_t = S_t^T C_t + D x_t
//
// The recurrence runs token by token in the order of the sequence whatever the cut, and both kernels for it (the one below, and the one of
// scan_columns.cuh for steps that bring many tokens) add up y in one order, so a position's result does not depend on how the prompt was cut
// into steps nor on what else is in the batch. Columns of S (one value dimension p each) are independent: a block takes 32 columns of one head of
// one request.
#include <climits>

#include "scan_columns.cuh"

// ---------------------------------------------------------------------------------------------- convolution
// out[t, c] = silu(bias[c] + sum_j w[c, j] * in[t - (taps-1-j), c]); inputs before the step's first token come from the
// request's tail (oldest first), which is zero for a new request.
template <typename T>
__global__ void causal_conv_silu_kernel(T* __restrict__ out, const T* __restrict__ proj, int proj_stride, int col0, int channels, int taps,
                                        const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state,
                                        long long slot_stride, const int* __restrict__ req_of_token, const int* __restrict__ cu_q,
                                        const int* __restrict__ state_slots) {
    pdl_wait();
    pdl_trigger();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (c >= channels) return;
    const int r = req_of_token[t];
    const int i = t - cu_q[r];
    const float* tail = state + (long long)state_slots[r] * slot_stride + (long long)c * (taps - 1);
    float acc = bias[c];
    for (int j = 0; j < taps; ++j) {
        const int back = taps - 1 - j;
        const float v = (i - back >= 0) ? Num<T>::to_f32(proj[(size_t)(t - back) * proj_stride + col0 + c]) : tail[taps - 1 + (i - back)];
        acc = fmaf(w[c * taps + j], v, acc);
    }
    out[(size_t)t * channels + c] = Num<T>::from_f32(acc / (1.f + expf(-acc)));
}

// Four taps on bf16 rows of whole 16-byte words: a thread takes eight channels of CONV_RUN tokens, one word a token, and keeps the last three inputs and the
// weights in registers. Element by element the kernel above fetched every input four times and its weight row 16 bytes apart: 2,048 tokens of
// 10,240 channels took 131 to 142 us, 56 to 62 a word at a time, 47 to 52 here (reading and writing each value once takes 13 us). The arithmetic is that of the kernel above, entry by entry.
constexpr int CONV_RUN = 16, CONV_THREADS = 128, CONV_AHEAD = 4;
__device__ __forceinline__ void conv_widen(const uint4& w, float (&v)[8]) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
__global__ void __launch_bounds__(CONV_THREADS) causal_conv4_silu_words_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ proj, int proj_stride,
                                                                               int col0, int channels, int n_tokens, const float* __restrict__ w,
                                                                               const float* __restrict__ bias, const float* __restrict__ state,
                                                                               long long slot_stride, const int* __restrict__ req_of_token,
                                                                               const int* __restrict__ cu_q, const int* __restrict__ state_slots) {
    pdl_wait();
    pdl_trigger();
    const int c = (blockIdx.x * CONV_THREADS + threadIdx.x) * 8;
    if (c >= channels) return;
    float wt[8][4], b[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float4 x = *reinterpret_cast<const float4*>(w + (size_t)(c + e) * 4);
        wt[e][0] = x.x; wt[e][1] = x.y; wt[e][2] = x.z; wt[e][3] = x.w;
        b[e] = bias[c + e];
    }
    const int first = blockIdx.y * CONV_RUN, last = min(first + CONV_RUN, n_tokens);
    float past[3][8];      // the inputs of the tokens three, two and one back
    int r = -1;
    for (int t0 = first; t0 < last; t0 += CONV_AHEAD) {
        uint4 words[CONV_AHEAD];       // asked for together: one behind the other's request, each waited for its trip to memory
        int requests[CONV_AHEAD];
#pragma unroll
        for (int k = 0; k < CONV_AHEAD; ++k) {
            const int t = min(t0 + k, last - 1);
            words[k] = *reinterpret_cast<const uint4*>(proj + (size_t)t * proj_stride + col0 + c);
            requests[k] = req_of_token[t];
        }
#pragma unroll
        for (int k = 0; k < CONV_AHEAD; ++k) {
            const int t = t0 + k;
            if (t >= last) break;
            if (requests[k] != r) {     // the run's first token or a request's: what lies before it comes from the rows before, or from the request's tail
                r = requests[k];
                const int i = t - cu_q[r];
                const float* tail = state + (long long)state_slots[r] * slot_stride + (long long)c * 3;
#pragma unroll
                for (int back = 3; back >= 1; --back) {
                    if (i - back >= 0) conv_widen(*reinterpret_cast<const uint4*>(proj + (size_t)(t - back) * proj_stride + col0 + c), past[3 - back]);
                    else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) past[3 - back][e] = tail[e * 3 + 3 + (i - back)];
                    }
                }
            }
            float now[8], o[8];
            conv_widen(words[k], now);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float acc = fmaf(wt[e][0], past[0][e], b[e]);
                acc = fmaf(wt[e][1], past[1][e], acc);
                acc = fmaf(wt[e][2], past[2][e], acc);
                acc = fmaf(wt[e][3], now[e], acc);
                o[e] = acc / (1.f + expf(-acc));
                past[0][e] = past[1][e]; past[1][e] = past[2][e]; past[2][e] = now[e];
            }
            uint4 word;
            __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&word);
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = __floats2bfloat162_rn(o[2 * e], o[2 * e + 1]);
            *reinterpret_cast<uint4*>(out + (size_t)t * channels + c) = word;
        }
    }
}

// After the convolution read it: the tail becomes the last taps-1 inputs of (old tail ++ the step's inputs).
template <typename T>
__global__ void conv_tail_roll_kernel(float* __restrict__ state, long long slot_stride, const T* __restrict__ proj, int proj_stride, int col0,
                                      int channels, int taps, const int* __restrict__ cu_q, const int* __restrict__ state_slots) {
    pdl_wait();
    pdl_trigger();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (c >= channels) return;
    const int t0 = cu_q[r], q = cu_q[r + 1] - t0, keep = taps - 1;
    if (q <= 0) return;
    float* tail = state + (long long)state_slots[r] * slot_stride + (long long)c * keep;
    for (int k = 0; k < keep; ++k) {       // entry k reads entry k + q (not yet overwritten) or a new input
        const int src = q + k - keep;
        tail[k] = src >= 0 ? Num<T>::to_f32(proj[(size_t)(t0 + src) * proj_stride + col0 + c]) : tail[k + q];
    }
}

// ---------------------------------------------------------------------------------------------- recurrence
// grid (ceil(vdim / 32), heads, requests); block = 32 * NW threads with NW = ceil(N / 32). Lane l owns the value column
// p = 32 blockIdx.x + l, warp w the state entries 4 (w + NW m) .. + 3 for m = 0 .. 7, so a thread keeps 32 entries of S in registers and
// updates them with plain multiply-adds in pairs: B and C of a token are the same for all lanes and come from shared memory as
// broadcast 16-byte loads, no shuffles. The step's tokens go through shared memory TT at a time (B, C, x, softplus and decay,
// each computed once per token and block; the next tile is fetched while this one is computed); the warps' partial sums of y
// meet there too. Every NW-th four entries to a warp, so that a thread's sums are the first ones of the order in scan_columns.cuh.
// S is stored [heads, N, vdim]: the lanes of a warp read and write 128 contiguous bytes per state entry.
// The bound on registers: a step of single tokens is the state's way through them, and three blocks of four warps on an SM are what it took before.
template <typename T, int NW, int TT>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 3 : 1) ssm_scan_kernel(
    float* __restrict__ y, const T* __restrict__ xbc, const T* __restrict__ proj, int proj_stride, int dt_col0, int heads, int vdim, int N,
    int groups, const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip, float* __restrict__ state,
    long long slot_stride, const int* __restrict__ cu_q, const int* __restrict__ state_slots, int most) {
    constexpr int NP = 32 * NW;                       // N rounded up to whole warps
    extern __shared__ __align__(16) float scan_smem[];
    float* Bs = scan_smem;                            // [TT][NP]
    float* Cs = Bs + TT * NP;                         // [TT][NP]
    float* xs = Cs + TT * NP;                         // [TT][32]
    float* part = xs + TT * 32;                       // [TT][NW][32]
    float* dts = part + TT * NW * 32;                 // [TT]
    float* decays = dts + TT;                         // [TT]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p0 = blockIdx.x * 32, p = p0 + lane, h = blockIdx.y, r = blockIdx.z;
    const int t0 = cu_q[r], t1 = cu_q[r + 1];
    if (t1 <= t0 || t1 - t0 > most) return;          // requests of more tokens are the other kernel's of this step
    const int inner = heads * vdim, channels = inner + 2 * groups * N, g = h / (heads / groups);
    const int b_col = inner + g * N, c_col = inner + groups * N + g * N;
    float* S = state + (long long)state_slots[r] * slot_stride + (long long)h * N * vdim;
    f32x2 s[16];                                      // pair i: entries entry(i) and entry(i) + 1
    auto entry = [&](int i) { return 4 * (warp + NW * (i >> 1)) + 2 * (i & 1); };
    auto stored = [&](int e) { return (e < N && p < vdim) ? S[(size_t)e * vdim + p] : 0.f; };
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = pack2(stored(entry(i)), stored(entry(i) + 1));
    const float neg_a = -expf(a_log[h]), bias = dt_bias[h], skip = d_skip[h];

    // A tile's inputs are fetched into registers while the tile before it is computed (all loads of a tile are issued back to
    // back: one trip to memory per tile, hidden behind the sums), then written to shared memory between two barriers.
    constexpr int XPT = (TT + NW - 1) / NW;           // x values per thread and tile
    const int n = threadIdx.x;                        // this thread's state entry in the fetch (NP threads, NP entries)
    T bv[TT], cv[TT], xv[XPT], dtv = Num<T>::from_f32(0.f);
    auto fetch = [&](int tile) {
        const int nt = min(TT, t1 - tile);
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            const bool ok = t < nt && n < N;
            const T* row = xbc + (size_t)(tile + (t < nt ? t : 0)) * channels;
            bv[t] = ok ? row[b_col + n] : Num<T>::from_f32(0.f);
            cv[t] = ok ? row[c_col + n] : Num<T>::from_f32(0.f);
        }
#pragma unroll
        for (int j = 0; j < XPT; ++j) {
            const int i = threadIdx.x + j * 32 * NW, t = i >> 5, c = i & 31;
            xv[j] = (t < nt && p0 + c < vdim) ? xbc[(size_t)(tile + t) * channels + h * vdim + p0 + c] : Num<T>::from_f32(0.f);
        }
        if ((int)threadIdx.x < nt) dtv = proj[(size_t)(tile + threadIdx.x) * proj_stride + dt_col0 + h];
    };
    auto stash = [&](int tile) {
        const int nt = min(TT, t1 - tile);
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            Bs[t * NP + n] = Num<T>::to_f32(bv[t]);
            Cs[t * NP + n] = Num<T>::to_f32(cv[t]);
        }
#pragma unroll
        for (int j = 0; j < XPT; ++j) {
            const int i = threadIdx.x + j * 32 * NW;
            if (i < TT * 32) xs[i] = Num<T>::to_f32(xv[j]);
        }
        if ((int)threadIdx.x < nt) {
            const float dt = scan_softplus(Num<T>::to_f32(dtv) + bias);
            dts[threadIdx.x] = dt;
            decays[threadIdx.x] = expf(neg_a * dt);
        }
    };
    fetch(t0);
    stash(t0);
    __syncthreads();
    for (int tile = t0; tile < t1; tile += TT) {
        const int nt = min(TT, t1 - tile);
        const bool more = tile + TT < t1;
        if (more) fetch(tile + TT);
        for (int t = 0; t < nt; ++t) {
            const float decay = decays[t], dx = dts[t] * xs[t * 32 + lane];
            const f32x2 decay2 = pack2(decay, decay), dx2 = pack2(dx, dx);
            float four[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(Bs + t * NP + entry(2 * m)), c = *reinterpret_cast<const ulonglong2*>(Cs + t * NP + entry(2 * m));
                s[2 * m] = fma2(decay2, s[2 * m], mul2(b.x, dx2));
                s[2 * m + 1] = fma2(decay2, s[2 * m + 1], mul2(b.y, dx2));
                four[m] = scan_sum_four(s[2 * m], s[2 * m + 1], c.x, c.y);
            }
            part[(t * NW + warp) * 32 + lane] = scan_halve<8>(four);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nt * 32; i += 32 * NW) {
            const int t = i >> 5, c = i & 31;
            if (p0 + c >= vdim) continue;
            float v[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) v[w] = part[(t * NW + w) * 32 + c];
            y[(size_t)(tile + t) * inner + h * vdim + p0 + c] = fmaf(skip, xs[i], scan_halve<NW>(v));
        }
        if (!more) break;
        __syncthreads();   // everyone has read this tile's buffers
        stash(tile + TT);
        __syncthreads();
    }
    if (p < vdim) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float lo, hi;
            unpack2(s[i], lo, hi);
            if (entry(i) < N) S[(size_t)entry(i) * vdim + p] = lo;
            if (entry(i) + 1 < N) S[(size_t)(entry(i) + 1) * vdim + p] = hi;
        }
    }
}

// ---------------------------------------------------------------------------------------------- gated grouped norm
// v = y * silu(z); out = v * rsqrt(mean over the part of v^2 + eps) * weight. grid (parts, tokens).
template <typename T>
__global__ void gated_group_norm_kernel(T* __restrict__ out, const float* __restrict__ y, const T* __restrict__ proj, int proj_stride, int z_col0,
                                        const float* __restrict__ weight, int inner, int part, float eps) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[32];
    const int t = blockIdx.y, lo = blockIdx.x * part;
    float ss = 0.f;
    for (int i = threadIdx.x; i < part; i += blockDim.x) {
        const float z = Num<T>::to_f32(proj[(size_t)t * proj_stride + z_col0 + lo + i]);
        const float v = y[(size_t)t * inner + lo + i] * (z / (1.f + expf(-z)));
        ss = fmaf(v, v, ss);
    }
    ss = block_sum(ss, red);
    const float inv = 1.f / sqrtf(ss / (float)part + eps);
    for (int i = threadIdx.x; i < part; i += blockDim.x) {
        const float z = Num<T>::to_f32(proj[(size_t)t * proj_stride + z_col0 + lo + i]);
        const float v = y[(size_t)t * inner + lo + i] * (z / (1.f + expf(-z)));
        out[(size_t)t * inner + lo + i] = Num<T>::from_f32(v * inv * weight[lo + i]);
    }
}

// The same on whole 16-byte words, eight entries a thread, each read once and kept in registers between the sum and the output: the kernel above reads y and z
// twice, an entry at a time, and works the silu out twice. 2,048 tokens x 8,192 in 8 parts: 75 -> 32 us (20 us of bytes).
__global__ void gated_group_norm_words_kernel(__nv_bfloat16* __restrict__ out, const float* __restrict__ y, const __nv_bfloat16* __restrict__ proj, int proj_stride,
                                              int z_col0, const float* __restrict__ weight, int inner, int part, float eps) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[32];
    const int t = blockIdx.y, at = blockIdx.x * part + 8 * threadIdx.x;
    const bool ok = 8 * (int)threadIdx.x < part;
    float v[8] = {};
    float ss = 0.f;
    if (ok) {
        float z[8];
        conv_widen(*reinterpret_cast<const uint4*>(proj + (size_t)t * proj_stride + z_col0 + at), z);
        const float4 a = *reinterpret_cast<const float4*>(y + (size_t)t * inner + at), b = *reinterpret_cast<const float4*>(y + (size_t)t * inner + at + 4);
        const float ye[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = ye[e] * (z[e] / (1.f + expf(-z[e])));
            ss = fmaf(v[e], v[e], ss);
        }
    }
    ss = block_sum(ss, red);
    const float inv = 1.f / sqrtf(ss / (float)part + eps);
    if (ok) {
        uint4 word;
        __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&word);
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = __floats2bfloat162_rn(v[2 * e] * inv * weight[at + 2 * e], v[2 * e + 1] * inv * weight[at + 2 * e + 1]);
        *reinterpret_cast<uint4*>(out + (size_t)t * inner + at) = word;
    }
}

// ---------------------------------------------------------------------------------------------- launchers
// proj: the in-projection's output [tokens, proj_stride], columns [z: inner | x, B, C: channels | dt: heads].
template <typename T>
static int mamba_conv(void* out, const void* proj, int n_tokens, int n_requests, int proj_stride, int col0, int channels, int taps,
                      const float* w, const float* bias, float* state, long long slot_stride, const int* req_of_token, const int* cu_q,
                      const int* state_slots, cudaStream_t stream) {
    // The 16-byte form wants whole words and work enough for a thread per eight channels of 16 tokens, behind the first token of each request (which brings a
    // tail to fetch, an entry at a time). 10,240 channels, us, the general form and this one: 150 tokens 22 and 26, 256 28 and 28, 320 32 and 28, 2,048 138
    // and 67; single tokens of 17, 48 and 256 requests 13 and 34, 17 and 38, 48 and 58; 48 of them beside 200, 300 and 400 tokens 32 and
    // 38, 38 and 38, 44 and 40. 5,120 channels: 200 tokens 20 and 26, 400 26 and 26, 600 32 and 28.
    const auto words = [](const void* p) { return (uintptr_t)p % 16 == 0; };
    if (sizeof(T) == 2 && taps == 4 && (long long)(n_tokens - n_requests) * channels >= 3000000 && channels % 8 == 0 && proj_stride % 8 == 0 && col0 % 8 == 0 && words(out) && words(proj) && words(w))
        oxr_launch_small(causal_conv4_silu_words_kernel, dim3((channels / 8 + CONV_THREADS - 1) / CONV_THREADS, (n_tokens + CONV_RUN - 1) / CONV_RUN), dim3(CONV_THREADS), 0, stream, 
            (__nv_bfloat16*)out, (const __nv_bfloat16*)proj, proj_stride, col0, channels, n_tokens, w, bias, state, slot_stride, req_of_token, cu_q, state_slots);
    else {
        dim3 grid((channels + 127) / 128, n_tokens);
        oxr_launch_small(causal_conv_silu_kernel<T>, dim3(grid), dim3(128), 0, stream, (T*)out, (const T*)proj, proj_stride, col0, channels, taps, w, bias, state, slot_stride,
                                                            req_of_token, cu_q, state_slots);
    }
    if (taps > 1) {
        dim3 grid2((channels + 127) / 128, n_requests);
        oxr_launch_small(conv_tail_roll_kernel<T>, dim3(grid2), dim3(128), 0, stream, state, slot_stride, (const T*)proj, proj_stride, col0, channels, taps, cu_q, state_slots);
    }
    return oxr_launch_status();
}

OXR_API int oxr_mamba_conv(void* out, const void* proj, int n_tokens, int n_requests, int proj_stride, int col0, int channels, int taps,
                           const float* w, const float* bias, float* state, long long slot_stride, const int* req_of_token, const int* cu_q,
                           const int* state_slots, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (channels <= 0 || taps < 1 || n_tokens > 65535 * 64 || n_requests > 65535) return OXR_BAD_ARGUMENT;
    if (n_tokens > 65535) return OXR_BAD_ARGUMENT;
    return dtype == 0 ? mamba_conv<float>(out, proj, n_tokens, n_requests, proj_stride, col0, channels, taps, w, bias, state, slot_stride, req_of_token,
                                          cu_q, state_slots, stream)
                      : mamba_conv<__nv_bfloat16>(out, proj, n_tokens, n_requests, proj_stride, col0, channels, taps, w, bias, state, slot_stride,
                                                  req_of_token, cu_q, state_slots, stream);
}

template <typename T, int NW>
static void mamba_scan(float* y, const void* xbc, const void* proj, int n_requests, int proj_stride, int dt_col0, int heads, int vdim, int N, int groups,
                       const float* dt_bias, const float* a_log, const float* d_skip, float* state, long long slot_stride, const int* cu_q,
                       const int* state_slots, int most, cudaStream_t stream) {
    constexpr int TT = NW <= 4 ? 16 : 8;
    constexpr size_t smem = (size_t)(TT * (2 * 32 * NW + 32 + NW * 32 + 2)) * sizeof(float);
    static_assert(smem <= 48 * 1024, "the tile fits the default shared memory");
    dim3 grid((vdim + 31) / 32, heads, n_requests);
    oxr_launch(ssm_scan_kernel<T, NW, TT>, dim3(grid), dim3(32 * NW), smem, stream, false, y, (const T*)xbc, (const T*)proj, proj_stride, dt_col0, heads, vdim, N, groups, dt_bias,
                                                                a_log, d_skip, state, slot_stride, cu_q, state_slots, most);
}

// n_long requests bring at least long_from tokens; long_list (host memory, may be null) names them, the longest first. They go to the kernel of
// scan_columns.cuh, where that takes the sizes, all others to the kernel above, in a launch of its own. Which kernel takes a request changes no result.
OXR_API int oxr_mamba_scan(float* y, const void* xbc, const void* proj, int n_requests, int proj_stride, int dt_col0, int heads, int vdim, int N, int groups,
                           const float* dt_bias, const float* a_log, const float* d_skip, float* state, long long slot_stride, const int* cu_q,
                           const int* state_slots, int dtype, const int* long_list, int n_long, int long_from, cudaStream_t stream) {
    if (n_requests <= 0) return 0;
    if (heads <= 0 || vdim <= 0 || N <= 0 || N > 256 || groups <= 0 || heads % groups || n_requests > 65535 || heads > 65535) return OXR_BAD_ARGUMENT;
    int most = INT_MAX;
    if (n_long > 0) {
        const size_t size = dtype == 0 ? 4 : 2;
        const int inner = heads * vdim;
        ScanArgs a = {};
        a.x = xbc; a.k = (const char*)xbc + inner * size; a.q = (const char*)xbc + (inner + groups * N) * size;
        a.stride = inner + 2 * groups * N; a.k_group = heads / groups; a.dt = (const char*)proj + dt_col0 * size; a.dt_stride = proj_stride;
        a.dt_bias = dt_bias; a.a_log = a_log; a.skip = d_skip; a.y = y; a.state = state; a.slot_stride = slot_stride; a.cu_q = cu_q; a.state_slots = state_slots;
        a.heads = heads; a.DV = vdim; a.n_requests = n_requests;
        a.least = n_long < n_requests ? long_from : 0;
        a.order = RequestOrder(long_list, n_long);
        if (dtype == 0 ? scan_fits<float>(a, N) : scan_fits<__nv_bfloat16>(a, N)) {
            const int rc = dtype == 0 ? scan_launch<float, false>(a, N, n_long, stream) : scan_launch<__nv_bfloat16, false>(a, N, n_long, stream);
            if (rc || n_long >= n_requests) return rc;
            most = long_from - 1;
        }
    }
    const int nw = (N + 31) / 32;
#define OXR_SCAN(NW) \
    (dtype == 0 ? mamba_scan<float, NW>(y, xbc, proj, n_requests, proj_stride, dt_col0, heads, vdim, N, groups, dt_bias, a_log, d_skip, state, \
                                        slot_stride, cu_q, state_slots, most, stream) \
                : mamba_scan<__nv_bfloat16, NW>(y, xbc, proj, n_requests, proj_stride, dt_col0, heads, vdim, N, groups, dt_bias, a_log, d_skip, state, \
                                                slot_stride, cu_q, state_slots, most, stream))
    switch (nw) {
        case 1: OXR_SCAN(1); break;
        case 2: OXR_SCAN(2); break;
        case 3: OXR_SCAN(3); break;
        case 4: OXR_SCAN(4); break;
        case 5: OXR_SCAN(5); break;
        case 6: OXR_SCAN(6); break;
        case 7: OXR_SCAN(7); break;
        default: OXR_SCAN(8); break;
    }
#undef OXR_SCAN
    return oxr_launch_status();
}

OXR_API int oxr_gated_group_norm(void* out, const float* y, const void* proj, int n_tokens, int proj_stride, int z_col0, const float* weight, int inner,
                                 int parts, float eps, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (inner <= 0 || parts <= 0 || inner % parts || n_tokens > 65535) return OXR_BAD_ARGUMENT;
    const int part = inner / parts;
    const int threads = part >= 1024 ? 256 : 128;
    dim3 grid(parts, n_tokens);
    const auto words = [](const void* p) { return (uintptr_t)p % 16 == 0; };
    if (dtype == 1 && part % 8 == 0 && part <= 8192 && proj_stride % 8 == 0 && z_col0 % 8 == 0 && words(out) && words(y) && words(proj)) {
        oxr_launch_small(gated_group_norm_words_kernel, dim3(grid), dim3((part / 8 + 31) / 32 * 32), 0, stream, (__nv_bfloat16*)out, y, (const __nv_bfloat16*)proj, proj_stride, z_col0, weight,
                                                                                     inner, part, eps);
        return oxr_launch_status();
    }
    if (dtype == 0) oxr_launch_small(gated_group_norm_kernel<float>, dim3(grid), dim3(threads), 0, stream, (float*)out, y, (const float*)proj, proj_stride, z_col0, weight, inner, part, eps);
    else oxr_launch_small(gated_group_norm_kernel<__nv_bfloat16>, dim3(grid), dim3(threads), 0, stream, (__nv_bfloat16*)out, y, (const __nv_bfloat16*)proj, proj_stride, z_col0, weight,
                                                                              inner, part, eps);
    return oxr_launch_status();
}
