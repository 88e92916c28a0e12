// The token-by-token recurrence that gated linear attention (gla.cu) and Mamba-2 (mamba.cu) share, for steps that bring many tokens of a request:
//
//   S_t = decay_t * S_(t-1) + k_t x_t^T          o_t = S_t^T q_t          S [DK, DV] per request and head, fp32
//
// with a decay per key entry (VECTOR) or one per token and head. Columns of S are independent. Token by token in the order of the sequence, and with one
// order of the sum S^T q in every kernel that takes these recurrences (this one with four or eight entries a lane, and the two for few tokens a
// request in gla.cu and mamba.cu): four neighbouring entries first, then the upper half of the fours onto the lower half until one is left. So a position's result has
// the same bits however a prompt was cut into steps and whatever else is in the batch.
//
// What bounds it: a thread that owns one column reads 4 bytes of k, q and decay from shared memory for every entry it updates, and shared memory returns
// 64 bytes a cycle to an SM's registers (measured), so the loads took several times as long as the multiply-adds they fed. Here a thread owns E = 4 or 8
// entries of FOUR columns, so that a word read is used four times: J = DK / E lanes share a group of four columns, lane j holds the entries 4 (j + J i) ..
// + 3, as pairs for the packed fp32 multiply-add (which issues every second cycle: it saves issue slots, not time on the pipe); k and q stay in the
// activations' type until they are in registers. The dot products of J / 8 tokens meet in one butterfly that halves their number with every
// step (lane j ends with number j / 2 of them). What is left is issue slots: about 100 (E = 4) or 157 (E = 8) a token and warp.
// Raw values come by cp.async, tiles of TT tokens, STAGES - 1 tiles ahead; one barrier per tile. 32 / E warps a block.
// 2,048 tokens on a B200, L2 flushed before: 16 heads of 128 x 256 with a decay per entry 402 us (one column a thread: 774); 128 heads of 128 x 64 with one per
// token 614 (705), prompts of 700 and 700 tokens 356 (506).
#pragma once

#include <type_traits>

#include "common.cuh"

typedef unsigned long long f32x2;      // two floats, the lower half first
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi)); return d; }
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// The sums of v[0 .. N - 1] over a group of 2 N neighbouring lanes, number j / 2 of them for lane j of the group: every step sends half of the
// numbers that are left to the lane N, N / 2, ... away and keeps the other half; the last step adds the two lanes of a pair.
template <int N> __device__ __forceinline__ float group_reduce(float (&v)[N], int lane) {
    if constexpr (N == 1) return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
    else {
        float half[N / 2];
        const bool up = (lane & N) != 0;       // this lane keeps the upper half of the numbers
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float send = up ? v[i] : v[N / 2 + i], keep = up ? v[N / 2 + i] : v[i];
            half[i] = keep + __shfl_xor_sync(0xffffffffu, send, N);
        }
        return group_reduce<N / 2>(half, lane);
    }
}

__device__ __forceinline__ float add_halves(f32x2 v) {
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}
// The first step of every sum S^T q: the products of four neighbouring entries (two pairs), the second pair's added to the first's, then the halves
__device__ __forceinline__ float scan_sum_four(f32x2 s01, f32x2 s23, f32x2 q01, f32x2 q23) {
    return add_halves(fma2(s23, q23, mul2(s01, q01)));
}

// The others: the upper half onto the lower until one is left (N a power of two; else one after the other, for sizes that one kernel alone takes)
template <int N> __device__ __forceinline__ float scan_halve(const float (&v)[N]) {
    if constexpr (N == 1) return v[0];
    else if constexpr (N % 2 == 0) {
        float half[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) half[i] = v[i] + v[N / 2 + i];
        return scan_halve<N / 2>(half);
    } else {
        float sum = v[0];
#pragma unroll
        for (int i = 1; i < N; ++i) sum += v[i];
        return sum;
    }
}

// The requests of a launch in the order of their blocks. Blocks start in the order of their index, and a recurrence runs as long as its longest request: started
// last, that one would run alone at the end. The host knows the lengths and names up to 32 requests, the longest first (an index out of the kernel's arguments
// is the same for a whole warp to the compiler too; ranking the lengths on the device cost the delta rule's chain of one prompt 2 %). Else all of the
// step, the last first: the scheduler puts portions of prompts behind the requests that decode.
constexpr int LISTED_MAX = 32;
struct RequestOrder {
    int n = 0;                       // 0: none named
    int r[LISTED_MAX];
    RequestOrder(const int* list, int count) {
        if (list == nullptr || count > LISTED_MAX) return;
        n = count;
        for (int i = 0; i < n; ++i) r[i] = list[i];
    }
    int blocks(int n_requests) const { return n > 0 ? n : n_requests; }
};
__device__ __forceinline__ int request_of(const RequestOrder& o, int n_blocks, int z) { return o.n > 0 ? o.r[z] : n_blocks - 1 - z; }

struct ScanArgs {
    const void *k, *q, *x;           // row 0, head 0: rows of `stride` entries, heads (or, k and q, groups of heads) side by side
    int stride, k_group;             // entries per row; heads that share a k and a q
    const float* decay;              // VECTOR: [tokens, heads * DK]
    const void* dt;                  // else: the logits of dt, row 0, head 0 (rows of dt_stride entries), its bias, log of the rate, the skip
    int dt_stride;
    const float *dt_bias, *a_log, *skip;
    float q_scale;
    float* y;                        // [tokens, heads * DV]
    float* state;                    // slot: [heads, DK, DV]
    long long slot_stride;
    const int *cu_q, *state_slots;
    int heads, DV, n_requests;
    int least;                       // of the launch's requests those of fewer tokens are the other kernel's
    RequestOrder order = {nullptr, 0};
};

constexpr int SCAN_TT = 8, SCAN_STAGES = 4;

template <typename T, int J, int E, bool VECTOR> struct ScanShape {
    static constexpr int WARPS = 32 / E, THREADS = 32 * WARPS, DK = E * J, GROUPS = 32 / J, COLS = WARPS * GROUPS * 4;
    static constexpr int KB = DK * (int)sizeof(T), AB = VECTOR ? DK * 4 : 0, XB = COLS * (int)sizeof(T), TOKEN = 2 * KB + AB + XB;   // bytes of a token
    static constexpr size_t SMEM = (size_t)SCAN_STAGES * SCAN_TT * TOKEN;
};

__device__ __forceinline__ float scan_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// The entries of a lane (as pairs) of a k, q or decay vector: 4 from `at` and, of eight, 4 from J * 4 entries further on
template <int J, int E> __device__ __forceinline__ void scan_entries(const float* at, f32x2 (&v)[E / 2]) {
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(at + 4 * J * i);
        v[2 * i] = a.x; v[2 * i + 1] = a.y;
    }
}
__device__ __forceinline__ f32x2 scan_widen(uint32_t two) { return pack2(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u)); }
template <int J, int E> __device__ __forceinline__ void scan_entries(const __nv_bfloat16* at, f32x2 (&v)[E / 2]) {
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
        const uint2 a = *reinterpret_cast<const uint2*>(at + 4 * J * i);
        v[2 * i] = scan_widen(a.x); v[2 * i + 1] = scan_widen(a.y);
    }
}
__device__ __forceinline__ void scan_four(const float* at, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(at);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void scan_four(const __nv_bfloat16* at, float (&v)[4]) {
    const uint2 a = *reinterpret_cast<const uint2*>(at);
    v[0] = __uint_as_float(a.x << 16); v[1] = __uint_as_float(a.x & 0xffff0000u);
    v[2] = __uint_as_float(a.y << 16); v[3] = __uint_as_float(a.y & 0xffff0000u);
}

// grid (ceil(DV / COLS), heads, requests of this launch). Row pieces are whole 16-byte words (scan_fits).
template <typename T, int J, int E, bool VECTOR>
__global__ void __launch_bounds__(ScanShape<T, J, E, VECTOR>::THREADS) column_scan_kernel(const ScanArgs a) {
    using Sh = ScanShape<T, J, E, VECTOR>;
    constexpr int TT = SCAN_TT, TPG = J / 8, P = E / 2, W = 16 / (int)sizeof(T);      // tokens whose sums meet in one butterfly; entries of a 16-byte word
    extern __shared__ __align__(16) unsigned char column_smem[];
    __shared__ float scalars[SCAN_STAGES][2][TT];                             // dt and decay of a token, where a token has one
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j = lane % J;
    const int h = blockIdx.y, r = request_of(a.order, gridDim.z, blockIdx.z);
    const int p0 = blockIdx.x * Sh::COLS, c0 = (warp * Sh::GROUPS + lane / J) * 4;   // this thread's first column of the block
    const int t0 = a.cu_q[r], t1 = a.cu_q[r + 1], DV = a.DV;
    if (t1 <= t0 || t1 - t0 < a.least) return;
    const int n_tiles = (t1 - t0 + TT - 1) / TT;
    const T* kp = (const T*)a.k + (size_t)(h / a.k_group) * Sh::DK;
    const T* qp = (const T*)a.q + (size_t)(h / a.k_group) * Sh::DK;
    const T* xp = (const T*)a.x + (size_t)h * DV + p0;
    const float* ap = VECTOR ? a.decay + (size_t)h * Sh::DK : nullptr;
    const T* dtp = VECTOR ? nullptr : (const T*)a.dt + h;
    float neg_a = 0.f, dt_bias = 0.f, skip = 0.f;
    if constexpr (!VECTOR) { neg_a = -expf(a.a_log[h]); dt_bias = a.dt_bias[h]; skip = a.skip[h]; }

    const int x_words = min(Sh::COLS, DV - p0) / W;      // beyond them lie columns that nobody stores
    auto fetch = [&](int tile) {
        if (tile < n_tiles) {
            const int first = t0 + tile * TT, nt = min(TT, t1 - first);
            const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(column_smem + (size_t)(tile % SCAN_STAGES) * TT * Sh::TOKEN);
            constexpr int KW = Sh::KB / 16, AW = Sh::AB / 16, XW = Sh::XB / 16, WORDS = 2 * KW + AW + XW;
            for (int i = tid; i < nt * WORDS; i += Sh::THREADS) {
                const int t = i / WORDS, w = i % WORDS;
                const char* src;
                if (w < KW) src = reinterpret_cast<const char*>(kp + (size_t)(first + t) * a.stride) + 16 * w;
                else if (w < 2 * KW) src = reinterpret_cast<const char*>(qp + (size_t)(first + t) * a.stride) + 16 * (w - KW);
                else if (VECTOR && w < 2 * KW + AW) src = reinterpret_cast<const char*>(ap + (size_t)(first + t) * a.heads * Sh::DK) + 16 * (w - 2 * KW);
                else {
                    if (w - 2 * KW - AW >= x_words) continue;
                    src = reinterpret_cast<const char*>(xp + (size_t)(first + t) * a.stride) + 16 * (w - 2 * KW - AW);
                }
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + t * Sh::TOKEN + 16 * w), "l"(src) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch_dt = [&](int tile) -> float {
        const int t = t0 + tile * TT + tid;
        return (!VECTOR && tid < TT && t < t1) ? Num<T>::to_f32(dtp[(size_t)t * a.dt_stride]) : 0.f;
    };
    auto put_dt = [&](int tile, float z) {
        if (!VECTOR && tid < TT) {
            const float dt = scan_softplus(z + dt_bias);
            scalars[tile % SCAN_STAGES][0][tid] = dt;
            scalars[tile % SCAN_STAGES][1][tid] = expf(neg_a * dt);
        }
    };
#pragma unroll
    for (int i = 0; i < SCAN_STAGES - 1; ++i) {
        fetch(i);
        put_dt(i, fetch_dt(i));
    }

    float* S = a.state + (long long)a.state_slots[r] * a.slot_stride + (long long)h * Sh::DK * DV + p0 + c0;
    const bool mine = p0 + c0 < DV;                       // DV is a multiple of 4: all four columns or none
    f32x2 s[4][P];                                        // [column][pair of entries]
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int e = 4 * (j + J * (i >> 1)) + 2 * (i & 1);
        const float4 u = mine ? *reinterpret_cast<const float4*>(S + (size_t)e * DV) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v = mine ? *reinterpret_cast<const float4*>(S + (size_t)(e + 1) * DV) : make_float4(0.f, 0.f, 0.f, 0.f);
        s[0][i] = pack2(u.x, v.x); s[1][i] = pack2(u.y, v.y); s[2][i] = pack2(u.z, v.z); s[3][i] = pack2(u.w, v.w);
    }
    const int my_tok = (j >> 1) >> 2, my_col = c0 + ((j >> 1) & 3);
    const bool writes = (j & 1) == 0 && p0 + my_col < DV;
    float* yp = a.y + (size_t)h * DV + p0 + my_col;
    const size_t y_stride = (size_t)a.heads * DV;

    for (int tile = 0; tile < n_tiles; ++tile) {
        asm volatile("cp.async.wait_group %0;" ::"n"(SCAN_STAGES - 2) : "memory");      // this tile's copies have arrived
        __syncthreads();                                                                   // everyone's; and the stage of the tile before is free
        fetch(tile + SCAN_STAGES - 1);
        const float dt_next = fetch_dt(tile + SCAN_STAGES - 1);
        const unsigned char* stage = column_smem + (size_t)(tile % SCAN_STAGES) * TT * Sh::TOKEN;
        const float* sc = scalars[tile % SCAN_STAGES][0];
        const int first = t0 + tile * TT, nt = min(TT, t1 - first);
        auto tokens = [&](auto whole) {
            constexpr bool WHOLE = decltype(whole)::value;
#pragma unroll
            for (int t = 0; t < TT; t += TPG) {
                if (!WHOLE && t >= nt) break;
                float d[4 * TPG];
#pragma unroll
                for (int k = 0; k < TPG; ++k) {
                    if (!WHOLE && t + k >= nt) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) d[4 * k + c] = 0.f;
                        continue;
                    }
                    const unsigned char* tok = stage + (t + k) * Sh::TOKEN;
                    f32x2 kk[P], qq[P], aa[P];
                    float x[4];
                    scan_entries<J, E>(reinterpret_cast<const T*>(tok) + 4 * j, kk);
                    scan_entries<J, E>(reinterpret_cast<const T*>(tok + Sh::KB) + 4 * j, qq);
                    scan_four(reinterpret_cast<const T*>(tok + 2 * Sh::KB + Sh::AB) + c0, x);
                    if constexpr (VECTOR) scan_entries<J, E>(reinterpret_cast<const float*>(tok + 2 * Sh::KB) + 4 * j, aa);
                    else {
                        const float dt = sc[t + k], decay = sc[TT + t + k];
                        const f32x2 both = pack2(decay, decay);
#pragma unroll
                        for (int i = 0; i < P; ++i) aa[i] = both;
#pragma unroll
                        for (int c = 0; c < 4; ++c) x[c] *= dt;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const f32x2 xx = pack2(x[c], x[c]);
                        if constexpr (E == 8 && !VECTOR) {
                            // the same sums, the first pairs of both fours before the second ones: 6 to 12 % less time (Mamba-2, 128 heads of 128 x 64, 3 prompts
                            // of 700 tokens: 569 and 508 us), where four entries a lane or a decay per entry take more
                            f32x2 pairs[2];
#pragma unroll
                            for (int half = 0; half < 2; ++half)
#pragma unroll
                                for (int i = half; i < P; i += 2) {
                                    s[c][i] = fma2(aa[i], s[c][i], mul2(kk[i], xx));
                                    pairs[i / 2] = half == 0 ? mul2(s[c][i], qq[i]) : fma2(s[c][i], qq[i], pairs[i / 2]);
                                }
                            d[4 * k + c] = add_halves(pairs[0]) + add_halves(pairs[1]);
                        } else {
                            float four[P / 2];
#pragma unroll
                            for (int i = 0; i < P; i += 2) {
                                s[c][i] = fma2(aa[i], s[c][i], mul2(kk[i], xx));
                                s[c][i + 1] = fma2(aa[i + 1], s[c][i + 1], mul2(kk[i + 1], xx));
                                four[i / 2] = scan_sum_four(s[c][i], s[c][i + 1], qq[i], qq[i + 1]);
                            }
                            d[4 * k + c] = four[0];
                            if constexpr (E == 8) d[4 * k + c] += four[1];
                        }
                    }
                }
                float o = group_reduce<4 * TPG>(d, lane);
                if (writes && (WHOLE || t + my_tok < nt)) {
                    if constexpr (VECTOR) o *= a.q_scale;
                    else o = fmaf(skip, Num<T>::to_f32(reinterpret_cast<const T*>(stage + (t + my_tok) * Sh::TOKEN + 2 * Sh::KB)[my_col]), o);
                    yp[(size_t)(first + t + my_tok) * y_stride] = o;
                }
            }
        };
        if (nt == TT) tokens(std::true_type{});
        else tokens(std::false_type{});
        put_dt(tile + SCAN_STAGES - 1, dt_next);      // its stage was last read in the tile before
    }
    if (mine) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int e = 4 * (j + J * (i >> 1)) + 2 * (i & 1);
            float4 u, v;
            unpack2(s[0][i], u.x, v.x);
            unpack2(s[1][i], u.y, v.y);
            unpack2(s[2][i], u.z, v.z);
            unpack2(s[3][i], u.w, v.w);
            *reinterpret_cast<float4*>(S + (size_t)e * DV) = u;
            *reinterpret_cast<float4*>(S + (size_t)(e + 1) * DV) = v;
        }
    }
}

// Whether the kernel takes these sizes: 64, 128 or 256 key entries, every row piece and every state row whole 16-byte words.
template <typename T>
inline bool scan_fits(const ScanArgs& a, int DK) {
    constexpr int W = 16 / (int)sizeof(T);
    const auto whole = [](const void* p) { return (uintptr_t)p % 16 == 0; };
    return (DK == 64 || DK == 128 || DK == 256) && a.DV % W == 0 && a.stride % W == 0 && a.slot_stride % 4 == 0 && whole(a.k) && whole(a.q) && whole(a.x) &&
           whole(a.decay) && whole(a.state);
}

template <typename T, int J, int E, bool VECTOR>
int scan_launch_j(const ScanArgs& a, cudaStream_t stream) {
    using Sh = ScanShape<T, J, E, VECTOR>;
    if constexpr (Sh::SMEM > 40 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(column_scan_kernel<T, J, E, VECTOR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM);
        if (e != cudaSuccess) return 1000 + (int)e;
    }
    oxr_launch(column_scan_kernel<T, J, E, VECTOR>, dim3((a.DV + Sh::COLS - 1) / Sh::COLS, a.heads, a.order.blocks(a.n_requests)), dim3(Sh::THREADS), Sh::SMEM, stream, false, a);
    return oxr_launch_status();
}
// Eight entries a lane where that makes warps enough to hide one another's latencies (a warp alone on its scheduler issues an instruction every 3.4
// cycles), else four: twice the warps, each with half the work and almost the same overhead. Measured on a B200 by the warps that eight entries make, four against
// eight, us: a decay per entry 512 (16 heads of 128 x 256, 2,048 tokens) 400 and 574, 1,024 (two prompts of 700) 218 and 251, 1,536 304 and 318, 2,048 402
// and 390, 8,192 (16 of 100) 226 and 200; one per token 512 (64 heads of 128 x 64, 2,048 tokens) 465 and 549, 1,024 (two of 700) 219 and 217, 1,536 299 and 277, 2,048
// 404 and 338.
// Only the n_long requests that this kernel takes count, and only they get blocks: one prompt beside 20 single tokens is one request's warps, and a grid with blocks for the
// others too, more than are resident at once, was dealt out with three of the prompt's blocks to an SM instead of one (1,200 tokens of gated linear
// attention alone 239 us, beside three single tokens 361).
template <typename T, bool VECTOR>
int scan_launch(const ScanArgs& a, int DK, int n_long, cudaStream_t stream) {
    const bool wide = (long long)a.heads * a.DV * DK / 1024 * n_long >= (VECTOR ? 2048 : 1536);
    if (DK == 256) return scan_launch_j<T, 32, 8, VECTOR>(a, stream);
    if (DK == 128) return wide ? scan_launch_j<T, 16, 8, VECTOR>(a, stream) : scan_launch_j<T, 32, 4, VECTOR>(a, stream);
    return wide ? scan_launch_j<T, 8, 8, VECTOR>(a, stream) : scan_launch_j<T, 16, 4, VECTOR>(a, stream);
}
