// Mixers that carry a state of fixed size from token to token: the short causal convolution, the gated delta rule with a
// decay per key channel, and the state-space recurrence with a decay per head. T is the storage type of the projections
// (float or bfloat16); decays, step sizes, gates, unit norms and the states themselves are 32-bit.
//
// A step's batch is ragged: request r owns the rows seq_starts[r] .. seq_starts[r + 1] - 1, and its state lives in row
// seq_slots[r] of the state tensor (zeroed by the step when the request's first token is among the rows). The same kernels
// run a prompt portion of any length and a single decoded token: the recurrences walk their rows in order, so a position's
// result does not depend on how the request was cut into steps.
#include <math.h>

#include "common.cuh"
#include "scan_sums.cuh"

namespace {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

constexpr int CONV_MAX_TAPS = 8;
constexpr int CONV_BATCH = 8;
constexpr int CONV_CHUNK = 32;   // tokens of one request that a block walks; at least CONV_MAX_TAPS - 1

// y[t, c] = act(bias[c] + sum_j w[c, j] * u[t - taps + 1 + j, c]) over the rows of each request, where u before the step's
// first row comes from state[slot][taps - 1 + t][c] (t < 0: the request's last taps - 1 inputs of earlier steps) and the
// state is then moved on by the step's rows. A thread owns a channel; only the block of a request's first chunk reads the
// old state and writes the new one, each thread its own channel, so nothing races.
// The inputs are asked for CONV_BATCH tokens at a time (one after the other a token cost a trip to memory: 2,048 tokens of 6,144 channels
// in bfloat16 45 us -> 37 us), and where a request's rows lie, which the host sent before the step's first kernel, before the wait.
template <typename T>
__global__ void __launch_bounds__(128) causal_conv_kernel(const T* __restrict__ z, int z_stride, int C, const float* __restrict__ w,
                                                          const float* __restrict__ bias, float* __restrict__ state,
                                                          const int* __restrict__ seq_starts, const int* __restrict__ seq_slots,
                                                          T* __restrict__ out, int out_stride, int taps, int act) {
    pdl_trigger();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    // everything is aligned to the most taps there may be: w8[j] belongs to the input CONV_MAX_TAPS - 1 - j tokens back
    constexpr int H = CONV_MAX_TAPS - 1;
    const int skip = CONV_MAX_TAPS - taps;
    float w8[CONV_MAX_TAPS];
    float b = 0.f;
    if (c < C) {
#pragma unroll
        for (int j = 0; j < CONV_MAX_TAPS; ++j) w8[j] = j >= skip ? w[(size_t)c * taps + j - skip] : 0.f;
        if (bias) b = bias[c];
    }
    const int r = blockIdx.z;
    const int s0 = seq_starts[r], L = seq_starts[r + 1] - s0;
    const int t0 = blockIdx.y * CONV_CHUNK;
    float* st = state + (size_t)seq_slots[r] * (taps - 1) * C + c;
    pdl_wait();
    if (c >= C || t0 >= L) return;
    // in[j], j < H: the H inputs before the batch's first token (those that no tap reads stay zero); then the batch's own
    float in[H + CONV_BATCH];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const int t = t0 - H + j;
        in[j] = 0.f;
        if (j >= skip) in[j] = t >= 0 ? to_f32(z[(size_t)(s0 + t) * z_stride + c]) : st[(size_t)(taps - 1 + t) * C];
    }
    if (L == 1) {   // a decoded token: nothing to run in batches, and its window moves on by one (6,144 channels, 64 requests: as part of a batch 9.2 us)
        const float u = to_f32(z[(size_t)s0 * z_stride + c]);
        float y = b;
#pragma unroll
        for (int j = 0; j < H; ++j)
            if (j >= skip) y = fmaf(w8[j], in[j], y);
        y = fmaf(w8[H], u, y);
        if (act == 1) y = silu_f(y);
        out[(size_t)s0 * out_stride + c] = from_f32<T>(y);
#pragma unroll
        for (int j = 0; j < H; ++j)
            if (j >= skip) st[(size_t)(j - skip) * C] = j + 1 < H ? in[j + 1] : u;
        return;
    }
    const int t1 = min(L, t0 + CONV_CHUNK);
    for (int t = t0; t < t1; t += CONV_BATCH) {
#pragma unroll
        for (int k = 0; k < CONV_BATCH; ++k) in[H + k] = t + k < t1 ? to_f32(z[(size_t)(s0 + t + k) * z_stride + c]) : 0.f;
#pragma unroll
        for (int k = 0; k < CONV_BATCH; ++k) {
            if (t + k < t1) {
                float y = b;
#pragma unroll
                for (int j = 0; j < CONV_MAX_TAPS; ++j)
                    if (j >= skip) y = fmaf(w8[j], in[k + j], y);
                if (act == 1) y = silu_f(y);
                out[(size_t)(s0 + t + k) * out_stride + c] = from_f32<T>(y);
            }
        }
        // the last H inputs so far (a short last batch keeps more of the older ones)
        const int n = min(CONV_BATCH, t1 - t);
        if (n == CONV_BATCH) {
#pragma unroll
            for (int j = 0; j < H; ++j) in[j] = in[j + CONV_BATCH];
        } else {
#pragma unroll
            for (int k = 0; k < CONV_BATCH; ++k)
                if (k < n) {
#pragma unroll
                    for (int j = 0; j < H + CONV_BATCH - 1; ++j) in[j] = in[j + 1];
                }
        }
    }
    if (t0 == 0) {
        if (t1 == L) {
#pragma unroll
            for (int j = 0; j < H; ++j)
                if (j >= skip) st[(size_t)(j - skip) * C] = in[j];
        } else {
            for (int i = 0; i < taps - 1; ++i) st[(size_t)i * C] = to_f32(z[(size_t)(s0 + L - (taps - 1) + i) * z_stride + c]);
        }
    }
}

// The same for steps with prompt portions, four taps and bfloat16, four neighbouring channels to a thread: 8-byte accesses (256 bytes a warp) where
// one channel to a thread moves 64, and eight tokens of them on their way. The result is rounded to bfloat16 (8 bits), so the exponential and the
// division are the fast 32-bit forms (errors of about 1e-7): the exact ones are half of this kernel's instructions. (6,144 channels, 2,048 tokens: 32 us with one
// channel to a thread, 27 with the exact forms.)
__global__ void __launch_bounds__(128) causal_conv4_kernel(const bf16* __restrict__ z, int z_stride, int C, const float* __restrict__ w,
                                                           const float* __restrict__ bias, float* __restrict__ state, const int* __restrict__ seq_starts,
                                                           const int* __restrict__ seq_slots, bf16* __restrict__ out, int out_stride, int act) {
    constexpr int TAPS = 4, H = TAPS - 1;
    pdl_trigger();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    float wt[TAPS][4], b[4] = {0.f, 0.f, 0.f, 0.f};   // [tap][channel]
    if (c < C) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float t[4];
            load4(w + (size_t)(c + i) * TAPS, t);
#pragma unroll
            for (int j = 0; j < TAPS; ++j) wt[j][i] = t[j];
        }
        if (bias) load4(bias + c, b);
    }
    const int r = blockIdx.z;
    const int s0 = seq_starts[r], L = seq_starts[r + 1] - s0;
    const int t0 = blockIdx.y * CONV_CHUNK;
    float* st = state + (size_t)seq_slots[r] * H * C + c;
    pdl_wait();
    if (c >= C || t0 >= L) return;
    const bf16* zr = z + (size_t)s0 * z_stride + c;
    bf16* o = out + (size_t)s0 * out_stride + c;
    float in[H + CONV_BATCH][4];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const int t = t0 - H + j;
        if (t >= 0) load4(zr + (size_t)t * z_stride, in[j]); else load4(st + (size_t)(H + t) * C, in[j]);
    }
    const int t1 = min(L, t0 + CONV_CHUNK);
    for (int t = t0; t < t1; t += CONV_BATCH) {
#pragma unroll
        for (int k = 0; k < CONV_BATCH; ++k)
            if (t + k < t1) load4(zr + (size_t)(t + k) * z_stride, in[H + k]);
#pragma unroll
        for (int k = 0; k < CONV_BATCH; ++k) {
            if (t + k < t1) {
                float y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    y[i] = b[i];
#pragma unroll
                    for (int j = 0; j < TAPS; ++j) y[i] = fmaf(wt[j][i], in[k + j][i], y[i]);
                    if (act == 1) y[i] = __fdividef(y[i], 1.0f + __expf(-y[i]));
                }
                store4(o + (size_t)(t + k) * out_stride, y);
            }
        }
        if (t + CONV_BATCH < t1) {
#pragma unroll
            for (int j = 0; j < H; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) in[j][i] = in[j + CONV_BATCH][i];
        }
    }
    if (t0 == 0) {   // the request's last inputs become its state; every read of the old one is this block's and behind it
        float last[H][4];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int t = L - H + i;
            if (t >= 0) load4(zr + (size_t)t * z_stride, last[i]); else load4(st + (size_t)(H + t) * C, last[i]);
        }
#pragma unroll
        for (int i = 0; i < H; ++i) store4(st + (size_t)i * C, last[i]);
    }
}

// ------------------------------------------------------------------------------------------------
// What the delta rule's recurrence reads, made from the projections in one parallel pass. One warp per (token, head):
//   decay[n, h, d] = exp(-exp(A_log[h]) * softplus(a[n, h, d] + dt_bias[h, d]))
//   (per_head: one decay per head, decay[n, h] = exp(-exp(A_log[h]) * softplus(a[n, h] + dt_bias[h])))
//   beta[n, h]     = sigmoid(b[n, h])
// and, by the first head of every key group g, the unit vectors
//   qn[n, g, :] = q / sqrt(sum q^2 + unit_eps) * q_scale,   kn[n, g, :] = k / sqrt(sum k^2 + unit_eps),   kq[n, g] = kn . qn
template <typename T>
__global__ void __launch_bounds__(128) delta_prepare_kernel(const T* __restrict__ qkv, int qkv_stride, int q_col, int k_col,
                                                            const T* __restrict__ a, int a_stride, const T* __restrict__ bsrc,
                                                            int b_stride, const float* __restrict__ A_log,
                                                            const float* __restrict__ dt_bias, float* __restrict__ qn,
                                                            float* __restrict__ kn, float* __restrict__ kq, float* __restrict__ decay,
                                                            float* __restrict__ beta, int N, int H, int G, int D, float q_scale,
                                                            float unit_eps, int per_head) {
    pdl_trigger();
    pdl_wait();
    const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (item >= N * H) return;
    const int n = item / H, h = item % H;
    const float rate = expf(A_log[h]);
    if (per_head) {
        if (lane == 0) decay[(size_t)n * H + h] = expf(-rate * softplus_f(to_f32(a[(size_t)n * a_stride + h]) + dt_bias[h]));
    } else {
        for (int d = lane; d < D; d += 32) {
            const float x = to_f32(a[(size_t)n * a_stride + h * D + d]) + dt_bias[h * D + d];
            decay[((size_t)n * H + h) * D + d] = expf(-rate * softplus_f(x));
        }
    }
    if (lane == 0) beta[(size_t)n * H + h] = sigmoid_f(to_f32(bsrc[(size_t)n * b_stride + h]));
    const int per = H / G;
    if (h % per == 0) {
        const int g = h / per;
        const T* qr = qkv + (size_t)n * qkv_stride + q_col + g * D;
        const T* kr = qkv + (size_t)n * qkv_stride + k_col + g * D;
        float sq = 0.f, sk = 0.f, dot = 0.f;
        for (int d = lane; d < D; d += 32) {
            const float qv = to_f32(qr[d]), kv = to_f32(kr[d]);
            sq = fmaf(qv, qv, sq); sk = fmaf(kv, kv, sk); dot = fmaf(qv, kv, dot);
        }
        sq = warp_sum(sq); sk = warp_sum(sk); dot = warp_sum(dot);
        const float fq = q_scale / sqrtf(sq + unit_eps), fk = 1.0f / sqrtf(sk + unit_eps);
        for (int d = lane; d < D; d += 32) {
            qn[((size_t)n * G + g) * D + d] = to_f32(qr[d]) * fq;
            kn[((size_t)n * G + g) * D + d] = to_f32(kr[d]) * fk;
        }
        if (lane == 0) kq[(size_t)n * G + g] = dot * fq * fk;
    }
}

// ------------------------------------------------------------------------------------------------
// How the recurrences are laid out. Per head the state S is [D, DV] (D: key channels or state size). Its columns are
// independent of one another, and within a column a token's work is a sum over D: PARTS lanes share a column, lane part j holding
// the entries d = 4 PARTS i + 4 j + c (c < 4) of CPL columns side by side in registers, in pairs for the packed
// multiply-add; a block is four warps. In memory a state is kept column by column ([DV][D]), so that a lane's entries are 16-byte
// pieces and a column's lanes read one contiguous run. Tokens arrive in tiles of SCAN_TILE through a two-stage ring in shared
// memory (the next tile lands while this one is worked on; rows padded with zeros to DMAX), and with them the block's
// columns of the token's own input. PARTS depends on D alone and with it the order of every sum, so a result does not depend on
// how many rows a step brings; CPL changes no sum, so it follows the number of columns of the step.
//
// A long walk is bound by what a token costs one warp: bytes from shared memory into registers (128 a cycle for the whole
// multiprocessor, however many lanes read the same address), multiply-adds, and for the delta rule, whose update needs the token's own
// sum, the chain multiply-adds -> shuffles -> update. So: few lanes to a column, several columns to a lane, the rows of the next
// token loaded while this one is worked on, no branch between the tokens of a full tile, and sums that only a token's output
// needs are not reduced token by token but PARTS of them at a time, each lane ending with one (parts_scatter). Measured (one
// request of 2,048 tokens, bfloat16), with 32 and 16 lanes to one column before: delta rule, 16 heads of 128 x 128, 744 -> 432 us;
// state space, 64 heads of 64 values and 128 states, 682 -> 320 us.
constexpr int SCAN_TILE = 16;
constexpr int SCAN_THREADS = 128;
constexpr int SCAN_ALONE_ROWS = 64;   // steps whose longest request brings this many rows launch the scans alone

// lanes per column: the delta rule (16 entries a lane and column: its chain is shortest with few shuffles) and the others (8 entries)
static inline __host__ __device__ constexpr int delta_parts(int dmax) { return dmax >= 256 ? 16 : (dmax >= 128 ? 8 : 4); }
static inline __host__ __device__ constexpr int scan_parts(int dmax) { return dmax >= 32 ? dmax / 8 : 4; }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// rows of `count` tokens, each D floats at src + (first + t) * stride, into dst[t][DMAX] (zeros beyond D)
template <int DMAX>
__device__ __forceinline__ void fetch_rows(float* dst, const float* __restrict__ src, size_t stride, int count, int D, bool vec) {
    constexpr int Q = DMAX / 4;
    for (int i = threadIdx.x; i < count * Q; i += SCAN_THREADS) {
        const int t = i / Q, d = (i % Q) * 4;
        float* o = dst + t * DMAX + d;
        const float* p = src + (size_t)t * stride + d;
        if (vec && d < D) {
            cp_async16(o, p);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] = d + c < D ? p[c] : 0.f;
        }
    }
}

// a lane's entries of its column of the state, from / to st[D] (the column's run in memory)
template <int DPL, int PARTS>
__device__ __forceinline__ void load_column(float* S, const float* st, int part, int D, bool live, bool vec) {
#pragma unroll
    for (int i = 0; i < DPL / 4; ++i) {
        const int d = 4 * PARTS * i + 4 * part;
        if (live && vec && d < D) {
            const float4 v = *reinterpret_cast<const float4*>(st + d);
            S[4 * i] = v.x; S[4 * i + 1] = v.y; S[4 * i + 2] = v.z; S[4 * i + 3] = v.w;
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) S[4 * i + c] = (live && d + c < D) ? st[d + c] : 0.f;
        }
    }
}
template <int DPL, int PARTS>
__device__ __forceinline__ void store_column(const float* S, float* st, int part, int D, bool vec) {
#pragma unroll
    for (int i = 0; i < DPL / 4; ++i) {
        const int d = 4 * PARTS * i + 4 * part;
        if (vec && d < D) {
            *reinterpret_cast<float4*>(st + d) = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (d + c < D) st[d + c] = S[4 * i + c];
        }
    }
}
template <int DPL, int PARTS>
__device__ __forceinline__ void load_column(float2* S, const float* st, int part, int D, bool live, bool vec) {
    float v[DPL];
    load_column<DPL, PARTS>(v, st, part, D, live, vec);
#pragma unroll
    for (int i = 0; i < DPL / 2; ++i) S[i] = make_float2(v[2 * i], v[2 * i + 1]);
}
template <int DPL, int PARTS>
__device__ __forceinline__ void store_column(const float2* S, float* st, int part, int D, bool vec) {
    float v[DPL];
#pragma unroll
    for (int i = 0; i < DPL / 2; ++i) { v[2 * i] = S[i].x; v[2 * i + 1] = S[i].y; }
    store_column<DPL, PARTS>(v, st, part, D, vec);
}

// four neighbouring elements as they are stored (taking them apart is left to their use, like converting them)
template <typename T> struct Four;
template <> struct Four<float> {
    float4 w;
    __device__ __forceinline__ void clear() { w = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const float* p) { w = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void set(int c, float x) { if (c == 0) w.x = x; else if (c == 1) w.y = x; else if (c == 2) w.z = x; else w.w = x; }
    __device__ __forceinline__ float get(int c) const { return c == 0 ? w.x : (c == 1 ? w.y : (c == 2 ? w.z : w.w)); }
};
template <> struct Four<bf16> {
    uint2 w;
    __device__ __forceinline__ void clear() { w = make_uint2(0u, 0u); }
    __device__ __forceinline__ void load(const bf16* p) { w = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void set(int c, bf16 x) {
        const uint32_t bits = (uint32_t)__bfloat16_as_ushort(x) << (16 * (c & 1));
        if (c < 2) w.x |= bits; else w.y |= bits;   // (after clear())
    }
    __device__ __forceinline__ float get(int c) const {
        const uint32_t t = c < 2 ? w.x : w.y;
        return __uint_as_float((c & 1) ? t & 0xffff0000u : t << 16);
    }
};

// The gated delta rule. For every token, in order:
//   S <- decay (.) S (row d by decay[d]);  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
// With S' = decay (.) S both products of a token are taken from S': r = S'^T k and S'^T q, and then o = S'^T q + u (k . q), the last
// factor coming with the token. SCALAR: the decay is one number per token and head (decay [N, H]) and comes with the token's other
// numbers instead of as a row of D.
template <typename T, int DMAX, int CPL, bool SCALAR>
__global__ void __launch_bounds__(SCAN_THREADS) delta_scan_kernel(const T* __restrict__ v, int v_stride, int v_col, const float* __restrict__ qn,
                                                                  const float* __restrict__ kn, const float* __restrict__ kq,
                                                                  const float* __restrict__ decay, const float* __restrict__ beta,
                                                                  float* __restrict__ state, const int* __restrict__ seq_starts,
                                                                  const int* __restrict__ seq_slots, float* __restrict__ out, int H, int G,
                                                                  int D, int DV) {
    constexpr int PARTS = delta_parts(DMAX), DPL = DMAX / PARTS, COLS = SCAN_THREADS / PARTS * CPL, P2 = DPL / 2, BATCH = PARTS / CPL;
    extern __shared__ __align__(16) float scan_smem[];
    float* k_s = scan_smem;                              // [2][SCAN_TILE][DMAX]
    float* q_s = k_s + 2 * SCAN_TILE * DMAX;
    float* g_s = q_s + 2 * SCAN_TILE * DMAX;
    float* beta_s = g_s + (SCALAR ? 0 : 2 * SCAN_TILE * DMAX);   // [2][SCAN_TILE]
    float* kq_s = beta_s + 2 * SCAN_TILE;
    float* g1_s = kq_s + 2 * SCAN_TILE;                  // [2][SCAN_TILE]: the decay where it is one number per token
    float* v_s = g1_s + 2 * SCAN_TILE;                   // [2][SCAN_TILE][COLS]
    pdl_wait();
    const int part = threadIdx.x % PARTS;
    const int my_col = threadIdx.x / PARTS * CPL;        // the first of the lane's CPL columns, within the block
    const int col = blockIdx.x * COLS + my_col;
    const int h = blockIdx.y, r = blockIdx.z;
    const int g = h / (H / G);
    const bool vec = (D & 3) == 0;
    const int s0 = seq_starts[r], s1 = seq_starts[r + 1];
    if (s1 - s0 < SCAN_TILE) pdl_trigger();   // (a short walk: the kernel behind may move in and set up; see the end)
    float* st = state + ((size_t)seq_slots[r] * H + h) * DV * D;
    float2 S[CPL][P2];
#pragma unroll
    for (int u = 0; u < CPL; ++u) load_column<DPL, PARTS>(S[u], st + (size_t)min(col + u, DV - 1) * D, part, D, col + u < DV, vec);
    auto fetch = [&](int base, int buf) {   // the rows of a tile: asynchronous copies
        const int count = min(SCAN_TILE, s1 - base);
        fetch_rows<DMAX>(k_s + buf * SCAN_TILE * DMAX, kn + ((size_t)base * G + g) * D, (size_t)G * D, count, D, vec);
        fetch_rows<DMAX>(q_s + buf * SCAN_TILE * DMAX, qn + ((size_t)base * G + g) * D, (size_t)G * D, count, D, vec);
        if constexpr (!SCALAR) fetch_rows<DMAX>(g_s + buf * SCAN_TILE * DMAX, decay + ((size_t)base * H + h) * D, (size_t)H * D, count, D, vec);
    };
    // A tile's numbers per token (beta, k . q) and the block's columns of v: loaded into registers a tile ahead, put into shared
    // memory before the tile's work. Thread i < SCAN_TILE holds token i's numbers; the threads from the end backwards hold v,
    // VPT values each.
    constexpr int VPT = (SCAN_TILE * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
    float pre_beta = 0.f, pre_kq = 0.f, pre_g = 1.f;
    T pre_v[VPT];   // (as they are stored: converted here, they would be waited for here)
    auto load_small = [&](int base) {
        const int count = min(SCAN_TILE, s1 - base);
        if (threadIdx.x < count) {
            pre_beta = beta[(size_t)(base + threadIdx.x) * H + h];
            pre_kq = kq[(size_t)(base + threadIdx.x) * G + g];
            if constexpr (SCALAR) pre_g = decay[(size_t)(base + threadIdx.x) * H + h];
        }
#pragma unroll
        for (int n = 0; n < VPT; ++n) {
            const int j = SCAN_THREADS - 1 - threadIdx.x + n * SCAN_THREADS;
            const int t = j / COLS, c = blockIdx.x * COLS + j % COLS;
            pre_v[n] = (j < count * COLS && c < DV) ? v[(size_t)(base + t) * v_stride + v_col + h * DV + c] : from_f32<T>(0.f);
        }
    };
    auto store_small = [&](int buf) {
        if (threadIdx.x < SCAN_TILE) {
            beta_s[buf * SCAN_TILE + threadIdx.x] = pre_beta;
            kq_s[buf * SCAN_TILE + threadIdx.x] = pre_kq;
            if constexpr (SCALAR) g1_s[buf * SCAN_TILE + threadIdx.x] = pre_g;
        }
#pragma unroll
        for (int n = 0; n < VPT; ++n) {
            const int j = SCAN_THREADS - 1 - threadIdx.x + n * SCAN_THREADS;
            if (j < SCAN_TILE * COLS) v_s[buf * SCAN_TILE * COLS + j] = to_f32(pre_v[n]);
        }
    };
    if (s0 < s1) {
        fetch(s0, 0);
        load_small(s0);
    }
    cp_commit();
    int buf = 0;
    for (int base = s0; base < s1; base += SCAN_TILE, buf ^= 1) {
        const int count = min(SCAN_TILE, s1 - base);
        store_small(buf);                      // (this stage's last readers passed the barrier of the tile between)
        cp_wait<0>();
        __syncthreads();                       // this tile is in shared memory, and everyone is done with the other stage
        if (base + SCAN_TILE < s1) {
            fetch(base + SCAN_TILE, buf ^ 1);
            load_small(base + SCAN_TILE);
        }
        cp_commit();
        const float* kb = k_s + buf * SCAN_TILE * DMAX + 4 * part;
        const float* qb = q_s + buf * SCAN_TILE * DMAX + 4 * part;
        const float* gb = g_s + buf * SCAN_TILE * DMAX + 4 * part;
        struct Row { float2 k[P2], q[P2], g[SCALAR ? 1 : P2]; };
        auto load_row = [&](int t, Row& w) {
#pragma unroll
            for (int i = 0; i < DPL / 4; ++i) {
                const float4 k4 = *reinterpret_cast<const float4*>(kb + t * DMAX + 4 * PARTS * i);
                const float4 q4 = *reinterpret_cast<const float4*>(qb + t * DMAX + 4 * PARTS * i);
                w.k[2 * i] = make_float2(k4.x, k4.y); w.k[2 * i + 1] = make_float2(k4.z, k4.w);
                w.q[2 * i] = make_float2(q4.x, q4.y); w.q[2 * i + 1] = make_float2(q4.z, q4.w);
                if constexpr (!SCALAR) {
                    const float4 g4 = *reinterpret_cast<const float4*>(gb + t * DMAX + 4 * PARTS * i);
                    w.g[2 * i] = make_float2(g4.x, g4.y); w.g[2 * i + 1] = make_float2(g4.z, g4.w);
                }
            }
            if constexpr (SCALAR) {
                const float g1 = g1_s[buf * SCAN_TILE + t];
                w.g[0] = make_float2(g1, g1);
            }
        };
        // one token: rq[u] is this lane's share of S'^T q, u_out[u] the update, of its columns
        auto token = [&](int t, const Row& w, float* rq, float* u_out) {
            const float bt = beta_s[buf * SCAN_TILE + t];
            float sk[CPL];
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                float2 a[2];
                a[0] = a[1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < P2; ++i) {
                    S[u][i] = mul2(S[u][i], w.g[SCALAR ? 0 : i]);
                    a[i & 1] = fma2(S[u][i], w.k[i], a[i & 1]);
                }
                sk[u] = (a[0].x + a[0].y) + (a[1].x + a[1].y);
            }
#pragma unroll
            for (int u = 0; u < CPL; ++u) sk[u] = parts_sum<PARTS>(sk[u]);
#pragma unroll
            for (int u = 0; u < CPL; ++u) {   // (needs nothing of the sums above: runs while they travel)
                float2 a[2];
                a[0] = a[1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < P2; ++i) a[i & 1] = fma2(S[u][i], w.q[i], a[i & 1]);
                rq[u] = (a[0].x + a[0].y) + (a[1].x + a[1].y);
            }
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                const float x = bt * (v_s[(buf * SCAN_TILE + t) * COLS + my_col + u] - sk[u]);
#pragma unroll
                for (int i = 0; i < P2; ++i) S[u][i] = fma2(w.k[i], make_float2(x, x), S[u][i]);
                u_out[u] = x;
            }
        };
        float* o = out + (size_t)base * H * DV + h * DV + col;
        if (count == SCAN_TILE) {
            const int my_t = part / CPL, my_u = part % CPL;   // the sum of a batch that this lane ends with
            Row now;
            load_row(0, now);
#pragma unroll
            for (int t0 = 0; t0 < SCAN_TILE; t0 += BATCH) {
                float rq[PARTS], u_mine = 0.f;
#pragma unroll
                for (int t = 0; t < BATCH; ++t) {
                    Row next;
                    if (t0 + t + 1 < SCAN_TILE) load_row(t0 + t + 1, next);
                    float u[CPL];
                    token(t0 + t, now, rq + t * CPL, u);
#pragma unroll
                    for (int c = 0; c < CPL; ++c)
                        if (part == t * CPL + c) u_mine = u[c];
                    now = next;
                }
                const float mine = parts_scatter<PARTS>(rq, part);
                if (col + my_u < DV) o[(size_t)(t0 + my_t) * H * DV + my_u] = fmaf(u_mine, kq_s[buf * SCAN_TILE + t0 + my_t], mine);
            }
        } else {
            for (int t = 0; t < count; ++t) {
                Row now;
                load_row(t, now);
                float rq[CPL], u[CPL];
                token(t, now, rq, u);
#pragma unroll
                for (int c = 0; c < CPL; ++c) {
                    const float sum = parts_sum<PARTS>(rq[c]);
                    if (col + c < DV && part == 0) o[(size_t)t * H * DV + c] = fmaf(u[c], kq_s[buf * SCAN_TILE + t], sum);
                }
            }
        }
    }
    cp_wait<0>();
    // Only now may the next kernel's blocks move in: they would wait for this kernel's end, and a multiprocessor full of
    // waiting warps slowed this kernel's own long walk by a third (measured).
    pdl_trigger();
#pragma unroll
    for (int u = 0; u < CPL; ++u)
        if (col + u < DV) store_column<DPL, PARTS>(S[u], st + (size_t)(col + u) * D, part, D, vec);
}

// ------------------------------------------------------------------------------------------------
// The state-space recurrence with one decay per head. Per head, S is [NS, DV]; for every token, in order:
//   dt = softplus(dt_raw + dt_bias[h]);  S <- exp(-exp(A_log[h]) dt) S + dt B x^T;  y = S^T C + D[h] x
// B and C belong to the head's group and come straight from the convolution's result (type T), so their tiles are filled with
// plain loads a tile ahead (four entries at a time where the rows allow it); step size and decay are computed as a tile is put into
// shared memory.
// FIXED: linear attention with a fixed decay per head, S <- decay[h] S + k v^T; y = S^T q. q, k and v stand in the places of C, B
// and x (a head of their own each: G = H), pass silu as they are loaded, and there are neither step sizes nor a skip; A_log holds
// the decays themselves.
template <typename T, int NMAX, int CPL, bool FIXED>
__global__ void __launch_bounds__(SCAN_THREADS) ssm_scan_kernel(const T* __restrict__ xbc, int x_stride, int x_col, int b_col, int c_col,
                                                                const T* __restrict__ dt_raw, int dt_stride, const float* __restrict__ A_log,
                                                                const float* __restrict__ dt_bias, const float* __restrict__ Dskip,
                                                                float* __restrict__ state, const int* __restrict__ seq_starts,
                                                                const int* __restrict__ seq_slots, float* __restrict__ out, int H, int G,
                                                                int NS, int DV) {
    constexpr int PARTS = scan_parts(NMAX), DPL = NMAX / PARTS, COLS = SCAN_THREADS / PARTS * CPL, P2 = DPL / 2, BATCH = PARTS / CPL;
    extern __shared__ __align__(16) float scan_smem[];
    float* b_s = scan_smem;                              // [2][SCAN_TILE][NMAX]
    float* c_s = b_s + 2 * SCAN_TILE * NMAX;
    float* a_s = c_s + 2 * SCAN_TILE * NMAX;             // [2][SCAN_TILE]
    float* dt_s = a_s + 2 * SCAN_TILE;
    float* x_s = dt_s + 2 * SCAN_TILE;                   // [2][SCAN_TILE][COLS]
    const int part = threadIdx.x % PARTS;
    const int my_col = threadIdx.x / PARTS * CPL;        // the first of the lane's CPL columns, within the block
    const int col = blockIdx.x * COLS + my_col;
    const int h = blockIdx.y, r = blockIdx.z;
    const int g = h / (H / G);
    const bool vec = (NS & 3) == 0;
    const float rate = FIXED ? A_log[h] : expf(A_log[h]), bias = FIXED ? 0.f : dt_bias[h], skip = FIXED ? 0.f : Dskip[h];
    pdl_wait();
    const int s0 = seq_starts[r], s1 = seq_starts[r + 1];
    if (s1 - s0 < SCAN_TILE) pdl_trigger();   // (a short walk: see the delta rule's kernel)
    float* st = state + ((size_t)seq_slots[r] * H + h) * DV * NS;
    float2 S[CPL][P2];
#pragma unroll
    for (int u = 0; u < CPL; ++u) load_column<DPL, PARTS>(S[u], st + (size_t)min(col + u, DV - 1) * NS, part, NS, col + u < DV, vec);
    // A tile (B and C of its tokens, step size and decay, the block's columns of x) is loaded into registers a tile ahead, as it is
    // stored (converted at once it would be waited for at once: half of the walk), and put into shared memory before the tile's work.
    constexpr int QPT = (SCAN_TILE * NMAX / 4 + SCAN_THREADS - 1) / SCAN_THREADS;
    constexpr int XPT = (SCAN_TILE * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
    const bool vec_in = vec && (x_stride & 3) == 0 && (b_col & 3) == 0 && (c_col & 3) == 0 && ((uintptr_t)xbc & (4 * sizeof(T) - 1)) == 0;
    Four<T> pre_b[QPT], pre_c[QPT];
    T pre_x[XPT], pre_dt = from_f32<T>(0.f);
    auto load_tile = [&](int base) {
        const int count = min(SCAN_TILE, s1 - base);
#pragma unroll
        for (int n = 0; n < QPT; ++n) {
            const int i = threadIdx.x + n * SCAN_THREADS;
            const int t = i / (NMAX / 4), d = i % (NMAX / 4) * 4;
            const T* row = xbc + (size_t)(base + t) * x_stride + g * NS + d;
            pre_b[n].clear();
            pre_c[n].clear();
            if (t < count && d < NS) {
                if (vec_in) {
                    pre_b[n].load(row + b_col);
                    pre_c[n].load(row + c_col);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (d + c < NS) { pre_b[n].set(c, row[b_col + c]); pre_c[n].set(c, row[c_col + c]); }
                }
            }
        }
        if (!FIXED && threadIdx.x < count) pre_dt = dt_raw[(size_t)(base + threadIdx.x) * dt_stride + h];
#pragma unroll
        for (int n = 0; n < XPT; ++n) {
            const int j = SCAN_THREADS - 1 - threadIdx.x + n * SCAN_THREADS;
            const int t = j / COLS, c = blockIdx.x * COLS + j % COLS;
            pre_x[n] = (j < count * COLS && c < DV) ? xbc[(size_t)(base + t) * x_stride + x_col + h * DV + c] : from_f32<T>(0.f);
        }
    };
    auto store_tile = [&](int buf, int count) {   // (tokens that are not there cost nothing: decoded tokens come one to a tile)
#pragma unroll
        for (int n = 0; n < QPT; ++n) {
            const int i = threadIdx.x + n * SCAN_THREADS;
            if (i < count * (NMAX / 4)) {
                float b4[4], c4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {   // (silu(0) = 0: the padding stays)
                    b4[c] = pre_b[n].get(c);
                    c4[c] = pre_c[n].get(c);
                    if constexpr (FIXED) { b4[c] = silu_f(b4[c]); c4[c] = silu_f(c4[c]); }
                }
                store4(b_s + buf * SCAN_TILE * NMAX + 4 * i, b4);
                store4(c_s + buf * SCAN_TILE * NMAX + 4 * i, c4);
            }
        }
        if (!FIXED && threadIdx.x < count) {
            const float dt = softplus_f(to_f32(pre_dt) + bias);
            dt_s[buf * SCAN_TILE + threadIdx.x] = dt;
            a_s[buf * SCAN_TILE + threadIdx.x] = expf(-rate * dt);
        }
#pragma unroll
        for (int n = 0; n < XPT; ++n) {
            const int j = SCAN_THREADS - 1 - threadIdx.x + n * SCAN_THREADS;
            if (j < count * COLS) x_s[buf * SCAN_TILE * COLS + j] = FIXED ? silu_f(to_f32(pre_x[n])) : to_f32(pre_x[n]);
        }
    };
    if (s0 < s1) load_tile(s0);
    int buf = 0;
    for (int base = s0; base < s1; base += SCAN_TILE, buf ^= 1) {
        const int count = min(SCAN_TILE, s1 - base);
        store_tile(buf, count);                       // (this stage's last readers passed the barrier of the tile between)
        __syncthreads();                       // this tile is in shared memory
        if (base + SCAN_TILE < s1) load_tile(base + SCAN_TILE);
        const float* bb = b_s + buf * SCAN_TILE * NMAX + 4 * part;
        const float* cb = c_s + buf * SCAN_TILE * NMAX + 4 * part;
        struct Row { float2 b[P2], c[P2]; };
        auto load_row = [&](int t, Row& w) {
#pragma unroll
            for (int i = 0; i < DPL / 4; ++i) {
                const float4 b4 = *reinterpret_cast<const float4*>(bb + t * NMAX + 4 * PARTS * i);
                const float4 c4 = *reinterpret_cast<const float4*>(cb + t * NMAX + 4 * PARTS * i);
                w.b[2 * i] = make_float2(b4.x, b4.y); w.b[2 * i + 1] = make_float2(b4.z, b4.w);
                w.c[2 * i] = make_float2(c4.x, c4.y); w.c[2 * i + 1] = make_float2(c4.z, c4.w);
            }
        };
        auto token = [&](int t, const Row& w, float* y) {   // y[u]: this lane's share of S^T C of its columns
            const float a = FIXED ? rate : a_s[buf * SCAN_TILE + t], dt = FIXED ? 1.f : dt_s[buf * SCAN_TILE + t];
            const float2 a2 = make_float2(a, a);
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                const float xv = x_s[(buf * SCAN_TILE + t) * COLS + my_col + u];
                const float in = FIXED ? xv : dt * xv;
                const float2 in2 = make_float2(in, in);
                float2 sum[2];
                sum[0] = sum[1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < P2; ++i) {
                    S[u][i] = fma2(a2, S[u][i], mul2(w.b[i], in2));
                    sum[i & 1] = fma2(S[u][i], w.c[i], sum[i & 1]);
                }
                y[u] = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            }
        };
        float* o = out + (size_t)base * H * DV + h * DV + col;
        auto put = [&](int t, int u, float y) {
            o[(size_t)t * H * DV + u] = FIXED ? y : fmaf(skip, x_s[(buf * SCAN_TILE + t) * COLS + my_col + u], y);
        };
        if (count == SCAN_TILE) {
            const int my_t = part / CPL, my_u = part % CPL;   // the sum of a batch that this lane ends with
            Row now;
            load_row(0, now);
#pragma unroll
            for (int t0 = 0; t0 < SCAN_TILE; t0 += BATCH) {
                float y[PARTS];
#pragma unroll
                for (int t = 0; t < BATCH; ++t) {
                    Row next;
                    if (t0 + t + 1 < SCAN_TILE) load_row(t0 + t + 1, next);
                    token(t0 + t, now, y + t * CPL);
                    now = next;
                }
                const float mine = parts_scatter<PARTS>(y, part);
                if (col + my_u < DV) put(t0 + my_t, my_u, mine);
            }
        } else {
            for (int t = 0; t < count; ++t) {
                Row now;
                load_row(t, now);
                float y[CPL];
                token(t, now, y);
#pragma unroll
                for (int u = 0; u < CPL; ++u) {
                    const float sum = parts_sum<PARTS>(y[u]);
                    if (col + u < DV && part == 0) put(t, u, sum);
                }
            }
        }
    }
    pdl_trigger();                             // (not before: see the delta rule's kernel)
#pragma unroll
    for (int u = 0; u < CPL; ++u)
        if (col + u < DV) store_column<DPL, PARTS>(S[u], st + (size_t)(col + u) * NS, part, NS, vec);
}

// ------------------------------------------------------------------------------------------------
// The selective scan with a state per channel and state index (the recurrence of Mamba). Per channel c, S[c] is NS numbers; for
// every token, in order:
//   dt = softplus(dt_raw[c] + dt_bias[c]);  S[c, n] <- exp(dt A[c, n]) S[c, n] + dt x[c] B[n];  y[c] = sum_n S[c, n] C[n] + D[c] x[c]
// with A = -exp(A_log) [C, NS], B and C shared by all channels of a token. The result leaves as y * silu(z) in the storage type.
// The layout is the one above with a channel in the place of a column: PARTS lanes share a channel, each with its entries of S and
// of A in registers; a block owns SCAN_THREADS / PARTS channels; tiles of SCAN_TILE tokens are loaded into registers a tile ahead.
// 2,048 channels, 16 states, eight prompts of 64 to 511 tokens (bfloat16), with step sizes waited for as they were loaded and a reduction per token before: 214 -> 105 us.
template <typename T, int NMAX, int PARTS, int TILE>
__global__ void __launch_bounds__(SCAN_THREADS) selective_scan_kernel(const T* __restrict__ x, int x_stride, const T* __restrict__ dt_raw, int dt_stride,
                                                                      const T* __restrict__ bc, int bc_stride, int b_col, int c_col,
                                                                      const T* __restrict__ z, int z_stride, const float* __restrict__ A_log,
                                                                      const float* __restrict__ dt_bias, const float* __restrict__ Dskip,
                                                                      float* __restrict__ state, const int* __restrict__ seq_starts,
                                                                      const int* __restrict__ seq_slots, T* __restrict__ out, int C, int NS) {
    constexpr int DPL = NMAX / PARTS, COLS = SCAN_THREADS / PARTS;
    constexpr bool WHOLE = TILE % PARTS == 0;   // a full tile's sums are added up PARTS at a time
    extern __shared__ __align__(16) float scan_smem[];
    float* b_s = scan_smem;                              // [2][TILE][NMAX]
    float* c_s = b_s + 2 * TILE * NMAX;
    float* x_s = c_s + 2 * TILE * NMAX;             // [2][TILE][COLS]
    float* dt_s = x_s + 2 * TILE * COLS;
    float* z_s = dt_s + 2 * TILE * COLS;
    const int part = threadIdx.x % PARTS;
    const int my_col = threadIdx.x / PARTS;
    const int col = blockIdx.x * COLS + my_col;
    const int r = blockIdx.z;
    const bool live = col < C;
    const bool vec = (NS & 3) == 0;
    // the channel's rates and numbers do not depend on the kernel before: fetched before the wait
    float A[DPL];
    load_column<DPL, PARTS>(A, A_log + (size_t)(live ? col : 0) * NS, part, NS, live, vec);
#pragma unroll
    for (int i = 0; i < DPL; ++i) A[i] = -expf(A[i]);
    const float skip = live ? Dskip[col] : 0.f;
    constexpr int BPT = (TILE * NMAX + SCAN_THREADS - 1) / SCAN_THREADS;
    constexpr int XPT = (TILE * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
    T pre_b[BPT], pre_c[BPT], pre_x[XPT], pre_dt[XPT], pre_z[XPT];   // (as they are stored: see above)
    // (a thread stages the same channel of the block in all its pieces: COLS divides the block)
    const int stage_c = blockIdx.x * COLS + threadIdx.x % COLS;
    pdl_wait();
    const float bias = stage_c < C ? dt_bias[stage_c] : 0.f;
    const int s0 = seq_starts[r], s1 = seq_starts[r + 1];
    if (s1 - s0 < SCAN_TILE) pdl_trigger();   // (a short walk: see the delta rule's kernel)
    float* st = state + ((size_t)seq_slots[r] * C + (live ? col : 0)) * NS;
    float S[DPL];
    load_column<DPL, PARTS>(S, st, part, NS, live, vec);
    auto load_tile = [&](int base) {
        const int count = min(TILE, s1 - base);
#pragma unroll
        for (int n = 0; n < BPT; ++n) {
            const int i = threadIdx.x + n * SCAN_THREADS;
            const int t = i / NMAX, d = i % NMAX;
            const bool in = t < count && d < NS;
            const size_t row = (size_t)(base + t) * bc_stride;
            pre_b[n] = in ? bc[row + b_col + d] : from_f32<T>(0.f);
            pre_c[n] = in ? bc[row + c_col + d] : from_f32<T>(0.f);
        }
#pragma unroll
        for (int n = 0; n < XPT; ++n) {
            const int j = threadIdx.x + n * SCAN_THREADS;
            const int t = j / COLS, c = blockIdx.x * COLS + j % COLS;
            const bool in = j < count * COLS && c < C;
            pre_x[n] = in ? x[(size_t)(base + t) * x_stride + c] : from_f32<T>(0.f);
            pre_z[n] = in ? z[(size_t)(base + t) * z_stride + c] : from_f32<T>(0.f);
            pre_dt[n] = in ? dt_raw[(size_t)(base + t) * dt_stride + c] : from_f32<T>(0.f);
        }
    };
    auto store_tile = [&](int buf, int count) {   // step sizes and gates are taken here, a tile behind their loads, which nobody waits for
#pragma unroll
        for (int n = 0; n < BPT; ++n) {
            const int i = threadIdx.x + n * SCAN_THREADS;
            if (i < count * NMAX) {
                b_s[buf * TILE * NMAX + i] = to_f32(pre_b[n]);
                c_s[buf * TILE * NMAX + i] = to_f32(pre_c[n]);
            }
        }
#pragma unroll
        for (int n = 0; n < XPT; ++n) {
            const int j = threadIdx.x + n * SCAN_THREADS;
            if (j < count * COLS) {
                x_s[buf * TILE * COLS + j] = to_f32(pre_x[n]);
                dt_s[buf * TILE * COLS + j] = softplus_f(to_f32(pre_dt[n]) + bias);
                z_s[buf * TILE * COLS + j] = silu_f(to_f32(pre_z[n]));
            }
        }
    };
    if (s0 < s1) load_tile(s0);
    int buf = 0;
    for (int base = s0; base < s1; base += TILE, buf ^= 1) {
        const int count = min(TILE, s1 - base);
        store_tile(buf, count);                       // (this stage's last readers passed the barrier of the tile between)
        __syncthreads();                       // this tile is in shared memory
        if (base + TILE < s1) load_tile(base + TILE);
        const float* bb = b_s + buf * TILE * NMAX + 4 * part;
        const float* cb = c_s + buf * TILE * NMAX + 4 * part;
        auto token = [&](int t) {   // returns this lane's share of the channel's sum
            const float xv = x_s[(buf * TILE + t) * COLS + my_col];
            const float dt = dt_s[(buf * TILE + t) * COLS + my_col];
            const float u = dt * xv;
            float y0 = 0.f, y1 = 0.f;
#pragma unroll
            for (int i = 0; i < DPL / 4; ++i) {
                const float4 b4 = *reinterpret_cast<const float4*>(bb + t * NMAX + 4 * PARTS * i);
                const float4 c4 = *reinterpret_cast<const float4*>(cb + t * NMAX + 4 * PARTS * i);
                float* sp = S + 4 * i;
                const float* ap = A + 4 * i;
                sp[0] = fmaf(expf(dt * ap[0]), sp[0], b4.x * u); sp[1] = fmaf(expf(dt * ap[1]), sp[1], b4.y * u);
                sp[2] = fmaf(expf(dt * ap[2]), sp[2], b4.z * u); sp[3] = fmaf(expf(dt * ap[3]), sp[3], b4.w * u);
                y0 = fmaf(sp[0], c4.x, y0); y1 = fmaf(sp[1], c4.y, y1); y0 = fmaf(sp[2], c4.z, y0); y1 = fmaf(sp[3], c4.w, y1);
            }
            return y0 + y1;
        };
        auto put = [&](int t, float y) {
            const int at = (buf * TILE + t) * COLS + my_col;
            out[(size_t)(base + t) * C + col] = from_f32<T>(fmaf(skip, x_s[at], y) * z_s[at]);
        };
        if (WHOLE && count == TILE) {
#pragma unroll
            for (int t0 = 0; t0 < TILE; t0 += PARTS) {
                float y[PARTS];
#pragma unroll
                for (int t = 0; t < PARTS; ++t) y[t] = token(t0 + t);
                const float mine = parts_scatter<PARTS>(y, part);
                if (live) put(t0 + part, mine);
            }
        } else {
            for (int t = 0; t < count; ++t) {
                const float y = parts_sum<PARTS>(token(t));
                if (live && part == 0) put(t, y);
            }
        }
    }
    pdl_trigger();                             // (not before: see the delta rule's kernel)
    if (live) store_column<DPL, PARTS>(S, st, part, NS, vec);
}

template <typename T>
int launch_conv(const T* z, int z_stride, int C, const float* w, const float* bias, float* state, const int* seq_starts,
                const int* seq_slots, T* out, int out_stride, int taps, int act, int R, int max_rows, cudaStream_t s) {
    const dim3 grid((C + 127) / 128, (max_rows + CONV_CHUNK - 1) / CONV_CHUNK, R);
    return launch_kernel(causal_conv_kernel<T>, grid, dim3(128), 0, s, z, z_stride, C, w, bias, state, seq_starts, seq_slots, out,
                         out_stride, taps, act);
}

// Several columns to a lane as soon as one each would be more warps than the device has schedulers: the step's columns decide (a lane
// with more of them makes each token longer, but reads the token's rows once for all).
static inline bool many_columns(long long columns, int parts) { return columns * parts > 148LL * SCAN_THREADS * 2; }
// (but not where a block would then be wider than the columns there are: its lanes beyond them idle)
static inline int padded(int columns, int block) { return (columns + block - 1) / block * block; }

template <typename T, int DM, int CPL, bool SCALAR>
int launch_delta_scan_one(const T* v, int v_stride, int v_col, const float* qn, const float* kn, const float* kq, const float* decay,
                          const float* beta, float* state, const int* seq_starts, const int* seq_slots, float* out, int H, int G, int D, int DV,
                          int R, bool alone, cudaStream_t s) {
    constexpr int cols = SCAN_THREADS / delta_parts(DM) * CPL;
    const dim3 grid((DV + cols - 1) / cols, H, R);
    const size_t smem = sizeof(float) * (2 * SCAN_TILE * ((SCALAR ? 2 : 3) * DM + 3 + cols));
    if (smem > 48 * 1024) cudaFuncSetAttribute(delta_scan_kernel<T, DM, CPL, SCALAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_kernel_on(alone, delta_scan_kernel<T, DM, CPL, SCALAR>, grid, dim3(SCAN_THREADS), smem, s, v, v_stride, v_col, qn, kn, kq, decay,
                            beta, state, seq_starts, seq_slots, out, H, G, D, DV);
}

template <typename T, int DM>
int launch_delta_scan_as(const T* v, int v_stride, int v_col, const float* qn, const float* kn, const float* kq, const float* decay,
                         const float* beta, float* state, const int* seq_starts, const int* seq_slots, float* out, int H, int G, int D, int DV,
                         int R, bool alone, bool scalar, cudaStream_t s) {
#define LLMIE_DELTA_ARGS v, v_stride, v_col, qn, kn, kq, decay, beta, state, seq_starts, seq_slots, out, H, G, D, DV, R, alone, s
    if (many_columns((long long)R * H * DV, delta_parts(DM)))
        return scalar ? launch_delta_scan_one<T, DM, 2, true>(LLMIE_DELTA_ARGS) : launch_delta_scan_one<T, DM, 2, false>(LLMIE_DELTA_ARGS);
    return scalar ? launch_delta_scan_one<T, DM, 1, true>(LLMIE_DELTA_ARGS) : launch_delta_scan_one<T, DM, 1, false>(LLMIE_DELTA_ARGS);
#undef LLMIE_DELTA_ARGS
}

template <typename T, int NM, int CPL, bool FIXED>
int launch_ssm_scan_one(const T* xbc, int x_stride, int x_col, int b_col, int c_col, const T* dt_raw, int dt_stride, const float* A_log,
                       const float* dt_bias, const float* Dskip, float* state, const int* seq_starts, const int* seq_slots, float* out, int H,
                       int G, int NS, int DV, int R, bool alone, cudaStream_t s) {
    constexpr int cols = SCAN_THREADS / scan_parts(NM) * CPL;
    const dim3 grid((DV + cols - 1) / cols, H, R);
    const size_t smem = sizeof(float) * (2 * SCAN_TILE * (2 * NM + 2 + cols));
    if (smem > 48 * 1024) cudaFuncSetAttribute(ssm_scan_kernel<T, NM, CPL, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_kernel_on(alone, ssm_scan_kernel<T, NM, CPL, FIXED>, grid, dim3(SCAN_THREADS), smem, s, xbc, x_stride, x_col, b_col, c_col, dt_raw,
                            dt_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, out, H, G, NS, DV);
}

template <typename T, int NM>
int launch_ssm_scan_as(const T* xbc, int x_stride, int x_col, int b_col, int c_col, const T* dt_raw, int dt_stride, const float* A_log,
                       const float* dt_bias, const float* Dskip, float* state, const int* seq_starts, const int* seq_slots, float* out, int H,
                       int G, int NS, int DV, int R, bool alone, cudaStream_t s) {
#define LLMIE_SSM_ARGS xbc, x_stride, x_col, b_col, c_col, dt_raw, dt_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, out, H, G, NS, DV, R, alone, s
    constexpr int one = SCAN_THREADS / scan_parts(NM);   // a block's columns with one to a lane
    const bool fixed = !dt_raw;                          // no step sizes: the fixed decays of linear attention
    if constexpr (NM <= 32) {
        if (padded(DV, one) < padded(DV, 2 * one) || (long long)R * H * DV * scan_parts(NM) <= 148LL * SCAN_THREADS)   // (or not even a block per multiprocessor)
            return fixed ? launch_ssm_scan_one<T, NM, 1, true>(LLMIE_SSM_ARGS) : launch_ssm_scan_one<T, NM, 1, false>(LLMIE_SSM_ARGS);
    }
    if (many_columns((long long)R * H * DV, scan_parts(NM)) && padded(DV, 4 * one) == padded(DV, 2 * one))
        return fixed ? launch_ssm_scan_one<T, NM, 4, true>(LLMIE_SSM_ARGS) : launch_ssm_scan_one<T, NM, 4, false>(LLMIE_SSM_ARGS);
    return fixed ? launch_ssm_scan_one<T, NM, 2, true>(LLMIE_SSM_ARGS) : launch_ssm_scan_one<T, NM, 2, false>(LLMIE_SSM_ARGS);
#undef LLMIE_SSM_ARGS
}

// the padded size (16, 32, 64, 128 or 256) picks the instantiation
#define LLMIE_SCAN_DISPATCH(FN, SIZE, ...)              \
    {                                                   \
        if (SIZE <= 16) return FN<T, 16>(__VA_ARGS__);   \
        if (SIZE <= 32) return FN<T, 32>(__VA_ARGS__);   \
        if (SIZE <= 64) return FN<T, 64>(__VA_ARGS__);   \
        if (SIZE <= 128) return FN<T, 128>(__VA_ARGS__); \
        return FN<T, 256>(__VA_ARGS__);                  \
    }

template <typename T>
int launch_delta_scan(const T* v, int v_stride, int v_col, const float* qn, const float* kn, const float* kq, const float* decay,
                      const float* beta, float* state, const int* seq_starts, const int* seq_slots, float* out, int H, int G, int D,
                      int DV, int R, bool alone, bool scalar, cudaStream_t s) {
    LLMIE_SCAN_DISPATCH(launch_delta_scan_as, D, v, v_stride, v_col, qn, kn, kq, decay, beta, state, seq_starts, seq_slots, out, H, G, D, DV, R, alone, scalar, s)
}

template <typename T>
int launch_ssm_scan(const T* xbc, int x_stride, int x_col, int b_col, int c_col, const T* dt_raw, int dt_stride, const float* A_log,
                    const float* dt_bias, const float* Dskip, float* state, const int* seq_starts, const int* seq_slots, float* out,
                    int H, int G, int NS, int DV, int R, bool alone, cudaStream_t s) {
    LLMIE_SCAN_DISPATCH(launch_ssm_scan_as, NS, xbc, x_stride, x_col, b_col, c_col, dt_raw, dt_stride, A_log, dt_bias, Dskip, state, seq_starts,
                        seq_slots, out, H, G, NS, DV, R, alone, s)
}

template <typename T, int NM, int PARTS, int TILE>
int launch_selective_scan_as(const T* x, int x_stride, const T* dt_raw, int dt_stride, const T* bc, int bc_stride, int b_col, int c_col, const T* z,
                             int z_stride, const float* A_log, const float* dt_bias, const float* Dskip, float* state, const int* seq_starts,
                             const int* seq_slots, T* out, int C, int NS, int R, bool alone, cudaStream_t s) {
    constexpr int cols = SCAN_THREADS / PARTS;
    const dim3 grid((C + cols - 1) / cols, 1, R);
    const size_t smem = sizeof(float) * (2 * TILE * (2 * NM + 3 * cols));
    if (smem > 48 * 1024) cudaFuncSetAttribute(selective_scan_kernel<T, NM, PARTS, TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_kernel_on(alone, selective_scan_kernel<T, NM, PARTS, TILE>, grid, dim3(SCAN_THREADS), smem, s, x, x_stride, dt_raw, dt_stride, bc, bc_stride,
                            b_col, c_col, z, z_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, out, C, NS);
}

constexpr long long SELECTIVE_FEW = 32768;
template <typename T>
int launch_selective_scan(const T* x, int x_stride, const T* dt_raw, int dt_stride, const T* bc, int bc_stride, int b_col, int c_col, const T* z,
                          int z_stride, const float* A_log, const float* dt_bias, const float* Dskip, float* state, const int* seq_starts,
                          const int* seq_slots, T* out, int C, int NS, int R, bool alone, bool short_rows, cudaStream_t s) {
#define LLMIE_SELECTIVE_ARGS x, x_stride, dt_raw, dt_stride, bc, bc_stride, b_col, c_col, z, z_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, out, C, NS, R, alone, s
    // (decoded tokens come one to a tile: a tile of SCAN_TILE would only take the room that more blocks at once need)
#define LLMIE_SELECTIVE(NM, PARTS) (short_rows ? launch_selective_scan_as<T, NM, PARTS, 4>(LLMIE_SELECTIVE_ARGS) : launch_selective_scan_as<T, NM, PARTS, SCAN_TILE>(LLMIE_SELECTIVE_ARGS))
    // An exponential per entry and token is most of the work, so a channel's entries are shared out among more lanes than a head's column would
    // be, the more the fewer channels there are (the model's sizes alone decide, never the batch: see scan_parts).
    const bool few = (long long)C * 16 <= SELECTIVE_FEW;
    if (NS <= 16) return LLMIE_SELECTIVE(16, 4);
    if (NS <= 32) return LLMIE_SELECTIVE(32, 8);
    if (NS <= 64) return few ? LLMIE_SELECTIVE(64, 16) : LLMIE_SELECTIVE(64, 8);
    if (NS <= 128) return few ? LLMIE_SELECTIVE(128, 16) : LLMIE_SELECTIVE(128, 8);
    return LLMIE_SELECTIVE(256, 16);
#undef LLMIE_SELECTIVE
#undef LLMIE_SELECTIVE_ARGS
}

}  // namespace

// z: columns 0 .. C - 1 of rows of z_stride elements (the caller offsets the pointer); state [slots][taps - 1][C] float.
LLMIE_API int llmie_causal_conv(const void* z, int z_stride, int C, const float* w, const float* bias, float* state,
                                const int* seq_starts, const int* seq_slots, void* out, int out_stride, int taps, int act, int R,
                                int max_rows, int dtype, cudaStream_t s) {
    if (R <= 0 || max_rows <= 0 || C <= 0) return 0;
    if (taps < 1 || taps > CONV_MAX_TAPS || R > 65535 || (max_rows + CONV_CHUNK - 1) / CONV_CHUNK > 65535 || act < 0 || act > 1)
        return LLMIE_ERR_BAD_ARGUMENT;
    if (dtype == DT_F32)
        return launch_conv<float>((const float*)z, z_stride, C, w, bias, state, seq_starts, seq_slots, (float*)out, out_stride, taps, act, R, max_rows, s);
    if (taps == 4 && max_rows > 1 && C % 4 == 0 && z_stride % 4 == 0 && out_stride % 4 == 0 && (((uintptr_t)z | (uintptr_t)out) & 7) == 0 &&
        (((uintptr_t)w | (uintptr_t)bias | (uintptr_t)state) & 15) == 0)
        return launch_kernel(causal_conv4_kernel, dim3((C / 4 + 127) / 128, (max_rows + CONV_CHUNK - 1) / CONV_CHUNK, R), dim3(128), 0, s, (const bf16*)z,
                             z_stride, C, w, bias, state, seq_starts, seq_slots, (bf16*)out, out_stride, act);
    return launch_conv<bf16>((const bf16*)z, z_stride, C, w, bias, state, seq_starts, seq_slots, (bf16*)out, out_stride, taps, act, R, max_rows, s);
}

LLMIE_API int llmie_delta_prepare(const void* qkv, int qkv_stride, int q_col, int k_col, const void* a, int a_stride, const void* b,
                                  int b_stride, const float* A_log, const float* dt_bias, float* qn, float* kn, float* kq, float* decay,
                                  float* beta, int N, int H, int G, int D, float q_scale, float unit_eps, int per_head, int dtype, cudaStream_t s) {
    if (N <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    const dim3 grid(((size_t)N * H + 3) / 4);
    if (dtype == DT_F32)
        return launch_kernel(delta_prepare_kernel<float>, grid, dim3(128), 0, s, (const float*)qkv, qkv_stride, q_col, k_col, (const float*)a,
                             a_stride, (const float*)b, b_stride, A_log, dt_bias, qn, kn, kq, decay, beta, N, H, G, D, q_scale, unit_eps, per_head);
    return launch_kernel(delta_prepare_kernel<bf16>, grid, dim3(128), 0, s, (const bf16*)qkv, qkv_stride, q_col, k_col, (const bf16*)a, a_stride,
                         (const bf16*)b, b_stride, A_log, dt_bias, qn, kn, kq, decay, beta, N, H, G, D, q_scale, unit_eps, per_head);
}

// state [slots][H][DV][D] float (column by column); out [N][H * DV] float; decay [N][H][D], or [N][H] with per_head
LLMIE_API int llmie_delta_scan(const void* v, int v_stride, int v_col, const float* qn, const float* kn, const float* kq,
                               const float* decay, const float* beta, float* state, const int* seq_starts, const int* seq_slots,
                               float* out, int H, int G, int D, int DV, int R, int max_rows, int per_head, int dtype, cudaStream_t s) {
    if (R <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || D > 256 || DV <= 0 || H > 65535 || R > 65535) return LLMIE_ERR_BAD_ARGUMENT;
    const bool alone = max_rows >= SCAN_ALONE_ROWS;   // a long walk: see launch_kernel_on
    if (dtype == DT_F32)
        return launch_delta_scan<float>((const float*)v, v_stride, v_col, qn, kn, kq, decay, beta, state, seq_starts, seq_slots, out, H, G, D, DV, R, alone, per_head != 0, s);
    return launch_delta_scan<bf16>((const bf16*)v, v_stride, v_col, qn, kn, kq, decay, beta, state, seq_starts, seq_slots, out, H, G, D, DV, R, alone, per_head != 0, s);
}

// state [slots][H][DV][NS] float (column by column); out [N][H * DV] float
LLMIE_API int llmie_ssm_scan(const void* xbc, int x_stride, int x_col, int b_col, int c_col, const void* dt_raw, int dt_stride,
                             const float* A_log, const float* dt_bias, const float* Dskip, float* state, const int* seq_starts,
                             const int* seq_slots, float* out, int H, int G, int NS, int DV, int R, int max_rows, int dtype, cudaStream_t s) {
    if (R <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || NS <= 0 || NS > 256 || DV <= 0 || H > 65535 || R > 65535 || !dt_raw) return LLMIE_ERR_BAD_ARGUMENT;
    const bool alone = max_rows >= SCAN_ALONE_ROWS;
    if (dtype == DT_F32)
        return launch_ssm_scan<float>((const float*)xbc, x_stride, x_col, b_col, c_col, (const float*)dt_raw, dt_stride, A_log, dt_bias, Dskip,
                                      state, seq_starts, seq_slots, out, H, G, NS, DV, R, alone, s);
    return launch_ssm_scan<bf16>((const bf16*)xbc, x_stride, x_col, b_col, c_col, (const bf16*)dt_raw, dt_stride, A_log, dt_bias, Dskip, state,
                                 seq_starts, seq_slots, out, H, G, NS, DV, R, alone, s);
}

// Linear attention with a fixed decay per head: z holds q and k (H heads of D columns from q_col, k_col) and v (H heads of DV from
// v_col), before silu; decay [H]; state [slots][H][DV][D] float (column by column); out [N][H * DV] float
LLMIE_API int llmie_linear_attention_scan(const void* z, int z_stride, int q_col, int k_col, int v_col, const float* decay, float* state,
                                          const int* seq_starts, const int* seq_slots, float* out, int H, int D, int DV, int R, int max_rows, int dtype,
                                          cudaStream_t s) {
    if (R <= 0) return 0;
    if (H <= 0 || D <= 0 || D > 256 || DV <= 0 || H > 65535 || R > 65535) return LLMIE_ERR_BAD_ARGUMENT;
    const bool alone = max_rows >= SCAN_ALONE_ROWS;
    if (dtype == DT_F32)
        return launch_ssm_scan<float>((const float*)z, z_stride, v_col, k_col, q_col, nullptr, 0, decay, nullptr, nullptr, state, seq_starts, seq_slots, out,
                                      H, H, D, DV, R, alone, s);
    return launch_ssm_scan<bf16>((const bf16*)z, z_stride, v_col, k_col, q_col, nullptr, 0, decay, nullptr, nullptr, state, seq_starts, seq_slots, out, H, H,
                                 D, DV, R, alone, s);
}

// x, dt_raw, z: [N] rows of C channels (the caller offsets the pointers to their first column); bc: rows that hold B from column
// b_col and C from column c_col (NS entries each); A_log [C][NS], dt_bias [C], Dskip [C]; state [slots][C][NS] float; out [N][C].
LLMIE_API int llmie_selective_scan(const void* x, int x_stride, const void* dt_raw, int dt_stride, const void* bc, int bc_stride, int b_col,
                                   int c_col, const void* z, int z_stride, const float* A_log, const float* dt_bias, const float* Dskip,
                                   float* state, const int* seq_starts, const int* seq_slots, void* out, int C, int NS, int R, int max_rows,
                                   int dtype, cudaStream_t s) {
    if (R <= 0) return 0;
    if (C <= 0 || NS <= 0 || NS > 256 || R > 65535) return LLMIE_ERR_BAD_ARGUMENT;
    const bool alone = max_rows >= SCAN_ALONE_ROWS;
    if (dtype == DT_F32)
        return launch_selective_scan<float>((const float*)x, x_stride, (const float*)dt_raw, dt_stride, (const float*)bc, bc_stride, b_col, c_col,
                                            (const float*)z, z_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, (float*)out, C, NS, R, alone, max_rows <= 4, s);
    return launch_selective_scan<bf16>((const bf16*)x, x_stride, (const bf16*)dt_raw, dt_stride, (const bf16*)bc, bc_stride, b_col, c_col,
                                       (const bf16*)z, z_stride, A_log, dt_bias, Dskip, state, seq_starts, seq_slots, (bf16*)out, C, NS, R, alone, max_rows <= 4, s);
}
