// Recurrences over long prompt portions, sixteen tokens at a time, in 32-bit arithmetic.
//
// All of them carry a matrix S [D, columns] per head, S_t = diag(a_t) S_(t-1) + k_t u_t^T, and put out S_t^T q_t:
//   KIND_DELTA_CHANNEL  the gated delta rule, a decay per key channel:  u_t = beta_t (v_t - (diag(a_t) S_(t-1))^T k_t)
//   KIND_DELTA_HEAD     the same with one decay per head
//   KIND_GIVEN          u_t = w_t v_t with a number w_t per token and head (state space: the step size)
// Written out over a chunk that starts from S_0, with G_t = a_1 ... a_t and every product entry by entry in d:
//   u_t = beta_t (v_t - S_0^T (G_t k_t) - sum_(s<t) A_ts u_s),   A_ts = sum_d k_t k_s a_(s+1) ... a_t      (delta rules)
//       = sum_(s<=t) T_ts v_s - S_0^T (sum_(s<=t) T_ts G_s k_s),     T = (1 + diag(beta) A)^-1 diag(beta)
//   o_t = S_0^T (G_t q_t) + sum_(s<=t) P_ts u_s,     P_ts = sum_d q_t k_s a_(s+1) ... a_t
//   S_16 = G_16 S_0 + sum_s (k_s a_(s+1) ... a_16) u_s^T
// so what goes from chunk to chunk are three small matrix products, and a token's chain (a product, a reduction, an update, 210 ns on one
// warp whatever else the multiprocessor could do) is a chunk's. T, P and the rows that meet S depend on no state: a prepare kernel makes them
// for all chunks side by side. No quotient of decays is taken: a_(s+1) ... a_t is split at the middle of the smallest aligned block that
// holds both tokens, into a factor of the later token and one of the earlier, both products of decays and at most 1, so nothing overflows
// however fast a state forgets.
//
// The scan: a block owns 16 columns of a head, its part of S in registers (a thread: one d, some columns) and a copy in shared memory that the
// products read. Phase 1, S_0^T (rows that meet S): each of eight warps takes a range of d and all 16 x 16 results, four tokens x two columns a
// lane, tokens in pairs for the packed multiply-add; the partial results meet in shared memory. Phase 2: the u, a token and column to a
// thread. Phase 3: outputs and the update of S. (With the substitution for u walked in the scan, a lane per column, the delta rule of 2,048
// tokens and 16 heads of 128 x 128 took 333 us with the prepare kernel; through T 302.) Rows are kept [d][16 tokens], four
// tokens in 16 bytes, the pieces of a row swapped by d so that the update's reads meet no bank twice; a chunk's rows are
// copied a chunk ahead.
//
// A chunk is bound by the bytes that go from shared memory into registers (128 a cycle, broadcast or not): about 3,100 of its 4,100 cycles; twice the
// warps with half the columns each move more of them and came out slower (229 -> 255 us). Measured in a step (us, token by token / prepare +
// scan): delta rule with channel decays, 2,048 tokens, 16 heads of 128 x 128, 430 / 64 + 229; state space, 64 heads of 64 values and 128
// states, 320 / 13 + 270. Eight prompts of 64 to 511 tokens and 8 heads (512 blocks, more than the device holds at once), 129 + 4 / 24 + 103.
//
// A request's results depend on where its steps cut it into chunks (in the last bits), so this form is for bfloat16 storage only, whose
// steps differ in their products' bits anyway; in float32 the token-by-token kernels keep every cut equal. Short portions stay there too.
#include <math.h>

#include "common.cuh"
#include "scan_sums.cuh"

namespace {

enum { KIND_DELTA_CHANNEL = 0, KIND_DELTA_HEAD = 1, KIND_GIVEN = 2 };

constexpr int CH = 16;           // tokens of a chunk
constexpr int COLS = 16;         // columns of a block
constexpr int SCAN_THREADS = 256;
constexpr int PAD = 20;          // floats between rows of 16 in shared memory

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Which chunk of the scratch arrays holds chunk i of request r: requests are given floor(first row / 16) + r onwards, which leaves none
// less room than it has chunks (N / 16 + R chunks in all).
__device__ __forceinline__ int chunk_slot(int first_row, int r, int i) { return first_row / CH + r + i; }
// Token piece j (four tokens) of row d lies at piece j ^ (d / 2 % 4): eight neighbouring d then cover all banks.
__device__ __forceinline__ int piece_at(int d, int j) { return (j ^ ((d >> 1) & 3)) * 4; }

// Scratch, in floats. Per chunk and head: the rows sum_s T_ts G_s k_s (delta rules) and, with channel decays, the rows G_t q_t and k_s a_(s+1) ...
// a_16, each [DMAX][16], and G_16 [DMAX]; then T and P [t][s] and the numbers, three rows of 16: w; G_t; a_(t+1) ... a_16 (the latter two where
// a decay is one number). Where it is, per chunk and group: the plain k and q rows.
template <int DMAX, int KIND> struct Layout {
    static constexpr int ROWS = DMAX * CH;
    static constexpr int SHARED_PART = KIND == KIND_DELTA_CHANNEL ? 0 : 2 * ROWS;                   // per chunk and group
    static constexpr int OWN_ROWS = KIND == KIND_DELTA_CHANNEL ? 3 * ROWS + DMAX : (KIND == KIND_DELTA_HEAD ? ROWS : 0);
    static constexpr int OWN = OWN_ROWS + (KIND == KIND_GIVEN ? 1 : 2) * CH * CH + 3 * CH;          // per chunk and head
    __host__ __device__ static size_t chunk(int H, int G) { return (size_t)G * SHARED_PART + (size_t)H * OWN; }
};

// Dot products of rows of DMAX floats (stride DMAX + 4): TP neighbouring threads to one dot, each a share of the 16-byte pieces.
template <int DMAX, int TP>
__device__ __forceinline__ float row_dot(const float* a, const float* b, int part) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
    for (int j = part; j < DMAX / 4; j += TP) {
        const float4 x = *reinterpret_cast<const float4*>(a + 4 * j), y = *reinterpret_cast<const float4*>(b + 4 * j);
        s0 = fmaf(x.x, y.x, s0); s1 = fmaf(x.y, y.y, s1); s0 = fmaf(x.z, y.z, s0); s1 = fmaf(x.w, y.w, s1);
    }
    s0 += s1;
#pragma unroll
    for (int o = TP / 2; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    return s0;
}

// a row [d][16 tokens] of a thread's own d, to global memory
__device__ __forceinline__ void put_row(float* to, int d, const float* v) {
#pragma unroll
    for (int j = 0; j < 4; ++j) store4(to + d * CH + piece_at(d, j), v + 4 * j);
}

// T from A [t][s] (s < t; the other entries are not read) and beta: a thread per column (16 threads), by substitution.
__device__ __forceinline__ void invert(const float* A, const float* beta, float* T) {
    const int j = threadIdx.x;
    float x[CH];
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < t; ++s) sum = s >= j ? fmaf(A[t * CH + s], x[s], sum) : sum;
        x[t] = t == j ? 1.f : (t > j ? -beta[t] * sum : 0.f);
    }
    const float b = beta[j];
#pragma unroll
    for (int t = 0; t < CH; ++t) T[t * CH + j] = x[t] * b;
}
// y[t] = sum_(s<=t) T[t][s] k[s] for a thread's own d
__device__ __forceinline__ void through(const float* T, const float* k, float* y) {
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s <= t; ++s) sum = fmaf(T[t * CH + s], k[s], sum);
        y[t] = sum;
    }
}

struct PrepareArgs {
    int z_stride, q_col, k_col;          // q and k of group g: columns q_col + g D, k_col + g D of z
    int a_stride, b_stride;              // decay logits and update logits (delta), step sizes (state space; b unused)
    const float *A_log, *dt_bias;        // per head (channel decays: dt_bias per head and channel)
    const int* seq_starts;
    float* scratch;
    int H, G, D;
    float q_scale, unit_eps;
};

// The unit vectors' factors and the dot of each token's own q and k: fq, fk, qk [16], from raw rows in shared memory (128 threads).
template <int DMAX>
__device__ __forceinline__ void unit_factors(const float* ks, const float* qs, float q_scale, float eps, float* fq, float* fk, float* qk) {
    const int t = threadIdx.x >> 3, part = threadIdx.x & 7;
    const float* k = ks + t * (DMAX + 4);
    const float* q = qs + t * (DMAX + 4);
    const float kk = row_dot<DMAX, 8>(k, k, part), qq = row_dot<DMAX, 8>(q, q, part), kq = row_dot<DMAX, 8>(q, k, part);
    if (part == 0) {
        const float a = q_scale / sqrtf(qq + eps), b = 1.0f / sqrtf(kk + eps);
        fq[t] = a; fk[t] = b; qk[t] = kq * a * b;
    }
}

// Block (i, h, r): chunk i of request r, head h; thread d < DMAX owns channel d. 128 threads.
template <typename T, int DMAX>
__global__ void __launch_bounds__(128) chunk_prepare_channel_kernel(const T* __restrict__ z, const T* __restrict__ a_raw, const T* __restrict__ b_raw,
                                                                    const __grid_constant__ PrepareArgs p) {
    using L = Layout<DMAX, KIND_DELTA_CHANNEL>;
    constexpr int RS = DMAX + 4;
    __shared__ __align__(16) float ks[CH * RS], qs[CH * RS];
    __shared__ float As[CH * CH], Ps[CH * CH], Ts[CH * CH], fq[CH], fk[CH], qk[CH], beta[CH];
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.z, h = blockIdx.y, i = blockIdx.x, d = threadIdx.x;
    const int s0 = p.seq_starts[r], first = s0 + i * CH, count = min(CH, p.seq_starts[r + 1] - first);
    if (count <= 0) return;
    const int g = h / (p.H / p.G);
    const bool live = d < p.D;
    float k[CH], q[CH], a[CH];
    const float rate = expf(p.A_log[h]), bias = live ? p.dt_bias[h * p.D + d] : 0.f;
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        k[t] = q[t] = 0.f;
        a[t] = 1.f;
        if (live && t < count) {
            const T* row = z + (size_t)(first + t) * p.z_stride + g * p.D + d;
            k[t] = to_f32(row[p.k_col]);
            q[t] = to_f32(row[p.q_col]);
            a[t] = to_f32(a_raw[(size_t)(first + t) * p.a_stride + h * p.D + d]);
        }
    }
    if (d < DMAX) {
#pragma unroll
        for (int t = 0; t < CH; ++t) { ks[t * RS + d] = k[t]; qs[t * RS + d] = q[t]; }
    }
    for (int e = threadIdx.x; e < CH * CH; e += 128) As[e] = Ps[e] = 0.f;
    if (threadIdx.x < CH) beta[threadIdx.x] = threadIdx.x < count ? sigmoid_f(to_f32(b_raw[(size_t)(first + threadIdx.x) * p.b_stride + h])) : 0.f;
#pragma unroll
    for (int t = 0; t < CH; ++t)
        if (live && t < count) a[t] = expf(-rate * softplus_f(a[t] + bias));
    __syncthreads();
    unit_factors<DMAX>(ks, qs, p.q_scale, p.unit_eps, fq, fk, qk);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < CH; ++t) { k[t] *= fk[t]; q[t] *= fq[t]; }
    // pairs whose smallest aligned block has B tokens: the later one in its second half, the earlier in its first
    auto level = [&](auto size) {
        constexpr int B = decltype(size)::value, HB = B / 2, PAIRS = CH * B / 4, TP = 128 / (2 * PAIRS);
        if (d < DMAX) {
#pragma unroll
            for (int b = 0; b < CH; b += B) {
                float f = 1.f;
#pragma unroll
                for (int s = b + HB - 1; s >= b; --s) { ks[s * RS + d] = k[s] * f; f *= a[s]; }
                f = 1.f;
#pragma unroll
                for (int t = b + HB; t < b + B; ++t) { f *= a[t]; ks[t * RS + d] = k[t] * f; qs[t * RS + d] = q[t] * f; }
            }
        }
        __syncthreads();
        const int dot = threadIdx.x / TP, part = threadIdx.x % TP, pair = dot % PAIRS, in = pair % (HB * HB), b = pair / (HB * HB) * B;
        const int t = b + HB + in / HB, s = b + in % HB;
        const bool second = dot >= PAIRS;
        const float sum = row_dot<DMAX, TP>((second ? qs : ks) + t * RS, ks + s * RS, part);
        if (part == 0) (second ? Ps : As)[t * CH + s] = sum;
        __syncthreads();
    };
    level(std::integral_constant<int, 16>{});
    level(std::integral_constant<int, 8>{});
    level(std::integral_constant<int, 4>{});
    level(std::integral_constant<int, 2>{});
    if (threadIdx.x < CH) invert(As, beta, Ts);
    __syncthreads();
    float* own = p.scratch + (size_t)chunk_slot(s0, r, i) * L::chunk(p.H, p.G) + (size_t)h * L::OWN;
    if (d < DMAX) {
        float y[CH];
        float f = 1.f;
#pragma unroll
        for (int t = CH - 1; t >= 0; --t) { y[t] = k[t] * f; f *= a[t]; }
        put_row(own + 2 * L::ROWS, d, y);
        f = 1.f;
#pragma unroll
        for (int t = 0; t < CH; ++t) { f *= a[t]; k[t] *= f; q[t] *= f; }
        put_row(own + L::ROWS, d, q);
        own[3 * L::ROWS + d] = f;
        through(Ts, k, y);
        put_row(own, d, y);
    }
    for (int e = threadIdx.x; e < CH * CH; e += 128) {
        own[L::OWN_ROWS + e] = Ts[e];
        own[L::OWN_ROWS + CH * CH + e] = e / CH == e % CH ? qk[e / CH] : Ps[e];
    }
}

// Block (i, g, r): chunk i of request r, key group g and its heads. 128 threads.
template <typename T, int DMAX, int KIND>
__global__ void __launch_bounds__(128) chunk_prepare_kernel(const T* __restrict__ z, const T* __restrict__ a_raw, const T* __restrict__ b_raw,
                                                            const __grid_constant__ PrepareArgs p) {
    using L = Layout<DMAX, KIND>;
    constexpr bool DELTA = KIND == KIND_DELTA_HEAD;
    constexpr int RS = DMAX + 4, MATS = DELTA ? 2 : 1;
    __shared__ __align__(16) float ks[CH * RS], qs[CH * RS];
    __shared__ float fq[CH], fk[CH], qk[CH], a[2][CH], w[2][CH], As[DELTA ? CH * CH : 1], Ts[DELTA ? CH * CH : 1];
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.z, g = blockIdx.y, i = blockIdx.x, d = threadIdx.x;
    const int s0 = p.seq_starts[r], first = s0 + i * CH, count = min(CH, p.seq_starts[r + 1] - first);
    if (count <= 0) return;
    float k[CH], q[CH];
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        k[t] = q[t] = 0.f;
        if (d < p.D && t < count) {
            const T* row = z + (size_t)(first + t) * p.z_stride + g * p.D + d;
            k[t] = to_f32(row[p.k_col]);
            q[t] = to_f32(row[p.q_col]);
        }
    }
    if constexpr (!DELTA) {
#pragma unroll
        for (int t = 0; t < CH; ++t) q[t] *= p.q_scale;
    }
    if (d < DMAX) {
#pragma unroll
        for (int t = 0; t < CH; ++t) { ks[t * RS + d] = k[t]; qs[t * RS + d] = q[t]; }
    }
    __syncthreads();
    float* chunk = p.scratch + (size_t)chunk_slot(s0, r, i) * L::chunk(p.H, p.G);
    float* mine = chunk + (size_t)g * L::SHARED_PART;
    if constexpr (DELTA) {
        unit_factors<DMAX>(ks, qs, p.q_scale, p.unit_eps, fq, fk, qk);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < CH; ++t) { k[t] *= fk[t]; q[t] *= fq[t]; }
    }
    if (d < DMAX) {
        put_row(mine, d, k);
        put_row(mine + L::ROWS, d, q);
    }
    // a thread's two pairs (t, s), from the rows as they came (unit vectors: times their factors)
    float kk[2], qkd[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = (threadIdx.x >> 4) + 8 * e, s = threadIdx.x & 15;
        kk[e] = qkd[e] = 0.f;
        if (s <= t) {
            qkd[e] = row_dot<DMAX, 1>(qs + t * RS, ks + s * RS, 0);
            if constexpr (DELTA) {
                qkd[e] *= fq[t] * fk[s];
                if (s < t) kk[e] = row_dot<DMAX, 1>(ks + t * RS, ks + s * RS, 0) * fk[t] * fk[s];
            }
        }
    }
    const int per = p.H / p.G;
    for (int j = 0; j < per; ++j) {
        const int h = g * per + j, buf = j & 1;
        if (threadIdx.x < CH) {
            const int t = threadIdx.x;
            float decay = 1.f, weight = 0.f;
            if (t < count) {
                const float dt = softplus_f(to_f32(a_raw[(size_t)(first + t) * p.a_stride + h]) + p.dt_bias[h]);
                decay = expf(-expf(p.A_log[h]) * dt);
                weight = DELTA ? sigmoid_f(to_f32(b_raw[(size_t)(first + t) * p.b_stride + h])) : dt;
            }
            a[buf][t] = decay;
            w[buf][t] = weight;
        }
        __syncthreads();
        float* own = chunk + (size_t)p.G * L::SHARED_PART + (size_t)h * L::OWN;
        float* mats = own + L::OWN_ROWS;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = (threadIdx.x >> 4) + 8 * e, s = threadIdx.x & 15;
            float f = 1.f;
            for (int x = s + 1; x <= t; ++x) f *= a[buf][x];
            if constexpr (DELTA) As[t * CH + s] = kk[e] * f;
            mats[(MATS - 1) * CH * CH + t * CH + s] = qkd[e] * f;
        }
        if constexpr (DELTA) {
            __syncthreads();
            if (threadIdx.x < CH) invert(As, w[buf], Ts);
            __syncthreads();
            for (int e = threadIdx.x; e < CH * CH; e += 128) mats[e] = Ts[e];
            if (d < DMAX) {
                float y[CH], kept[CH], f = 1.f;
#pragma unroll
                for (int t = 0; t < CH; ++t) { f *= a[buf][t]; kept[t] = k[t] * f; }
                through(Ts, kept, y);
                put_row(own, d, y);
            }
        }
        if (threadIdx.x < CH) {
            const int t = threadIdx.x;
            float before = 1.f, after = 1.f;
            for (int x = 0; x <= t; ++x) before *= a[buf][x];
            for (int x = CH - 1; x > t; --x) after *= a[buf][x];
            float* numbers = mats + MATS * CH * CH;
            numbers[t] = w[buf][t];
            numbers[CH + t] = before;
            numbers[2 * CH + t] = after;
        }
    }
}

template <typename T> struct ScanArgs {
    const float* scratch;
    const T* v;
    int v_stride, v_col;
    float* state;                // [slots, H, DV, D], column by column
    const int *seq_starts, *seq_slots;
    float* out;                  // [N, H, DV]
    const float* skip;           // [H] or null: out += skip v
    int H, G, D, DV;
};

// Block (x, h, r): 16 columns of head h of request r, all its chunks.
template <typename T, int DMAX, int KIND>
__global__ void __launch_bounds__(SCAN_THREADS) chunk_scan_kernel(const __grid_constant__ ScanArgs<T> p) {
    using L = Layout<DMAX, KIND>;
    constexpr bool DELTA = KIND != KIND_GIVEN, CHANNEL = KIND == KIND_DELTA_CHANNEL;
    constexpr int MATS = DELTA ? 2 : 1, WARPS = SCAN_THREADS / 32, DW = DMAX / WARPS, CT = COLS * DMAX / SCAN_THREADS;
    constexpr int STAGE = L::SHARED_PART + L::OWN;   // a stage: the group's rows, then the head's own
    extern __shared__ __align__(16) float sm[];
    float* S_s = sm + 2 * STAGE;                       // [DMAX][PAD]
    float* red = S_s + DMAX * PAD;                     // [WARPS][MATS][COLS][PAD]: a warp's share of the q (and k) rows' products
    float* vs = red + WARPS * MATS * COLS * PAD;       // [CH][COLS]: the chunk's values (delta rules)
    float* us = vs + CH * COLS;                        // [CH][COLS]
    float* us_end = us + CH * COLS;                    // the same, decayed to the chunk's end (one decay per head)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.y, r = blockIdx.z, col0 = blockIdx.x * COLS;
    const int s0 = p.seq_starts[r], s1 = p.seq_starts[r + 1];
    const int g = h / (p.H / p.G);
    const size_t chunk_floats = L::chunk(p.H, p.G);
    pdl_wait();
    const float* at = p.scratch + (size_t)chunk_slot(s0, r, 0) * chunk_floats;
    auto copy = [&](int i, int buf) {
        float* to = sm + buf * STAGE;
        const float* chunk = at + (size_t)i * chunk_floats;
        const float* own = chunk + (size_t)p.G * L::SHARED_PART + (size_t)h * L::OWN;
        if constexpr (!CHANNEL) {
            const float* rows = chunk + (size_t)g * L::SHARED_PART;
            for (int e = tid; e < L::SHARED_PART / 4; e += SCAN_THREADS) cp_async16(to + 4 * e, rows + 4 * e);
            to += L::SHARED_PART;
        }
        for (int e = tid; e < L::OWN / 4; e += SCAN_THREADS) cp_async16(to + 4 * e, own + 4 * e);
    };
    // the thread's part of S: row d, columns c0 .. c0 + CT
    const int d = tid % DMAX, c0 = tid / DMAX * CT;
    float* st = p.state + ((size_t)p.seq_slots[r] * p.H + h) * p.DV * p.D;
    float S[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) S[c] = (d < p.D && col0 + c0 + c < p.DV) ? st[(size_t)(col0 + c0 + c) * p.D + d] : 0.f;
    auto show = [&] {
#pragma unroll
        for (int c = 0; c < CT; c += 4) store4(S_s + d * PAD + c0 + c, S + c);
    };
    show();
    // the thread's token and column of the values and results
    const int t = tid >> 4, c = tid & 15, col = col0 + c;
    T pre_v = from_f32<T>(0.f);
    auto load_v = [&](int base) {
        pre_v = from_f32<T>(0.f);
        if (base + t < s1 && col < p.DV) pre_v = p.v[(size_t)(base + t) * p.v_stride + p.v_col + h * p.DV + col];
    };
    const float skip = p.skip ? p.skip[h] : 0.f;
    if (s0 < s1) {
        copy(0, 0);
        load_v(s0);
    }
    cp_commit();
    int buf = 0;
    for (int base = s0, i = 0; base < s1; base += CH, ++i, buf ^= 1) {
        cp_wait<0>();
        __syncthreads();   // the chunk's rows and S are in shared memory, everyone is done with the other stage
        const float v = to_f32(pre_v);
        if (base + CH < s1) {
            copy(i + 1, buf ^ 1);
            load_v(base + CH);
        }
        cp_commit();
        const float* stage = sm + buf * STAGE;
        const float* own = stage + L::SHARED_PART;
        const float* k_rows = own;                                        // (delta rules) what u takes from S
        const float* q_rows = CHANNEL ? own + L::ROWS : stage + L::ROWS;
        const float* end_rows = CHANNEL ? own + 2 * L::ROWS : stage;
        const float* weights = own + L::OWN_ROWS;   // T
        const float* P = weights + (MATS - 1) * CH * CH;
        const float* numbers = P + CH * CH;
        if constexpr (DELTA) vs[t * COLS + c] = base + t < s1 ? v : 0.f;
        // phase 1
        {
            const int tg = lane >> 3, cg = lane & 7;
            float2 x[2][2], y[2][2];   // [column][token pair]
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int n = 0; n < 2; ++n) x[u][n] = y[u][n] = make_float2(0.f, 0.f);
#pragma unroll
            for (int e = 0; e < DW; ++e) {
                const int dd = warp * DW + e;
                const float2 s2 = *reinterpret_cast<const float2*>(S_s + dd * PAD + 2 * cg);
                const float2 sa = make_float2(s2.x, s2.x), sb = make_float2(s2.y, s2.y);
                const int piece = dd * CH + piece_at(dd, tg);
                const float4 q4 = *reinterpret_cast<const float4*>(q_rows + piece);
                y[0][0] = fma2(sa, make_float2(q4.x, q4.y), y[0][0]); y[0][1] = fma2(sa, make_float2(q4.z, q4.w), y[0][1]);
                y[1][0] = fma2(sb, make_float2(q4.x, q4.y), y[1][0]); y[1][1] = fma2(sb, make_float2(q4.z, q4.w), y[1][1]);
                if constexpr (DELTA) {
                    const float4 k4 = *reinterpret_cast<const float4*>(k_rows + piece);
                    x[0][0] = fma2(sa, make_float2(k4.x, k4.y), x[0][0]); x[0][1] = fma2(sa, make_float2(k4.z, k4.w), x[0][1]);
                    x[1][0] = fma2(sb, make_float2(k4.x, k4.y), x[1][0]); x[1][1] = fma2(sb, make_float2(k4.z, k4.w), x[1][1]);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float* to = red + (warp * MATS * COLS + 2 * cg + u) * PAD + 4 * tg;
                *reinterpret_cast<float4*>(to) = make_float4(y[u][0].x, y[u][0].y, y[u][1].x, y[u][1].y);
                if constexpr (DELTA) *reinterpret_cast<float4*>(to + COLS * PAD) = make_float4(x[u][0].x, x[u][0].y, x[u][1].x, x[u][1].y);
            }
        }
        __syncthreads();
        float y = 0.f;
        {
            float x = 0.f;
#pragma unroll
            for (int e = 0; e < WARPS; ++e) {
                y += red[(e * MATS * COLS + c) * PAD + t];
                if constexpr (DELTA) x += red[((e * MATS + 1) * COLS + c) * PAD + t];
            }
            if constexpr (!CHANNEL) y *= numbers[CH + t];
            float u;
            if constexpr (DELTA) {   // (rows of tokens that are not there are zero, T's too; of later tokens nothing, not even zero times an infinity)
                float u0 = -x, u1 = 0.f;
#pragma unroll
                for (int j = 0; j < CH / 4; ++j) {
                    const float4 t4 = *reinterpret_cast<const float4*>(weights + t * CH + 4 * j);
                    const float* v4 = vs + 4 * j * COLS + c;
                    u0 = fmaf(t4.x, 4 * j <= t ? v4[0] : 0.f, u0); u1 = fmaf(t4.y, 4 * j + 1 <= t ? v4[COLS] : 0.f, u1);
                    u0 = fmaf(t4.z, 4 * j + 2 <= t ? v4[2 * COLS] : 0.f, u0); u1 = fmaf(t4.w, 4 * j + 3 <= t ? v4[3 * COLS] : 0.f, u1);
                }
                u = u0 + u1;
            } else {
                u = numbers[t] * v;
            }
            if (base + t >= s1) u = 0.f;   // (a column that holds an infinity must not spread it through tokens that are not there)
            us[t * COLS + c] = u;
            if constexpr (!CHANNEL) us_end[t * COLS + c] = numbers[2 * CH + t] * u;
        }
        __syncthreads();
        // phase 3
        {
            float o0 = y, o1 = 0.f;
#pragma unroll
            for (int j = 0; j < CH / 4; ++j) {
                const float4 p4 = *reinterpret_cast<const float4*>(P + t * CH + 4 * j);
                const float* u4 = us + 4 * j * COLS + c;   // (of later tokens nothing, not even zero times an infinity)
                o0 = fmaf(p4.x, 4 * j <= t ? u4[0] : 0.f, o0); o1 = fmaf(p4.y, 4 * j + 1 <= t ? u4[COLS] : 0.f, o1);
                o0 = fmaf(p4.z, 4 * j + 2 <= t ? u4[2 * COLS] : 0.f, o0); o1 = fmaf(p4.w, 4 * j + 3 <= t ? u4[3 * COLS] : 0.f, o1);
            }
            if (base + t < s1 && col < p.DV) p.out[((size_t)(base + t) * p.H + h) * p.DV + col] = fmaf(skip, v, o0 + o1);
        }
        const float keep = CHANNEL ? own[3 * L::ROWS + d] : numbers[CH + CH - 1];
        float2 S2[CT / 2];
#pragma unroll
        for (int n = 0; n < CT / 2; ++n) S2[n] = mul2(make_float2(S[2 * n], S[2 * n + 1]), make_float2(keep, keep));
        const float* u_rows = CHANNEL ? us : us_end;
#pragma unroll
        for (int j = 0; j < CH / 4; ++j) {
            float k4[4];
            load4(end_rows + d * CH + piece_at(d, j), k4);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const float2 kd = make_float2(k4[n], k4[n]);
#pragma unroll
                for (int m = 0; m < CT / 4; ++m) {
                    const float4 u4 = *reinterpret_cast<const float4*>(u_rows + (4 * j + n) * COLS + c0 + 4 * m);
                    S2[2 * m] = fma2(kd, make_float2(u4.x, u4.y), S2[2 * m]);
                    S2[2 * m + 1] = fma2(kd, make_float2(u4.z, u4.w), S2[2 * m + 1]);
                }
            }
        }
#pragma unroll
        for (int n = 0; n < CT / 2; ++n) { S[2 * n] = S2[n].x; S[2 * n + 1] = S2[n].y; }
        show();
    }
    cp_wait<0>();
    pdl_trigger();
    if (s0 < s1) {
#pragma unroll
        for (int e = 0; e < CT; ++e)
            if (d < p.D && col0 + c0 + e < p.DV) st[(size_t)(col0 + c0 + e) * p.D + d] = S[e];
    }
}

template <typename T, int DMAX, int KIND>
int run_chunks(const T* z, const T* a, const T* b, const PrepareArgs& pa, const ScanArgs<T>& sa, int R, int max_len, cudaStream_t s) {
    using L = Layout<DMAX, KIND>;
    constexpr int MATS = KIND == KIND_GIVEN ? 1 : 2;
    constexpr int smem = (2 * (L::SHARED_PART + L::OWN) + DMAX * PAD + SCAN_THREADS / 32 * MATS * COLS * PAD + 3 * CH * COLS) * 4;
    static OncePerDevice granted;
    int rc = grant_shared(granted, chunk_scan_kernel<T, DMAX, KIND>, smem);
    if (rc) return rc;
    const int chunks = (max_len + CH - 1) / CH;
    if constexpr (KIND == KIND_DELTA_CHANNEL)
        rc = launch_kernel(chunk_prepare_channel_kernel<T, DMAX>, dim3(chunks, pa.H, R), dim3(128), 0, s, z, a, b, pa);
    else
        rc = launch_kernel(chunk_prepare_kernel<T, DMAX, KIND>, dim3(chunks, pa.G, R), dim3(128), 0, s, z, a, b, pa);
    if (rc) return rc;
    return launch_kernel_on(true, chunk_scan_kernel<T, DMAX, KIND>, dim3((sa.DV + COLS - 1) / COLS, sa.H, R), dim3(SCAN_THREADS), smem, s, sa);
}

template <int KIND>
int run_kind(const bf16* z, const bf16* a, const bf16* b, const PrepareArgs& pa, const ScanArgs<bf16>& sa, int R, int max_len, cudaStream_t s) {
    if (pa.D <= 64) return run_chunks<bf16, 64, KIND>(z, a, b, pa, sa, R, max_len, s);
    return run_chunks<bf16, 128, KIND>(z, a, b, pa, sa, R, max_len, s);
}

bool sizes_fit(int H, int G, int D, int DV, int R, int max_len) {
    return H >= 1 && G >= 1 && H % G == 0 && H <= 65535 && D >= 1 && D <= 128 && DV >= 1 && R >= 1 && R <= 65535 && max_len >= 1;
}

}  // namespace

// How many floats of scratch a step of N rows and R requests takes; 0: these sizes are not built.
LLMIE_API long long llmie_chunk_scratch(int kind, int H, int G, int D, int N, int R) {
    if (!sizes_fit(H, G, D, 1, R, 1) || kind < 0 || kind > KIND_GIVEN) return 0;
    const long long chunks = N / CH + R;
    const bool wide = D > 64;
    if (kind == KIND_DELTA_CHANNEL) return chunks * (long long)(wide ? Layout<128, 0>::chunk(H, G) : Layout<64, 0>::chunk(H, G));
    if (kind == KIND_DELTA_HEAD) return chunks * (long long)(wide ? Layout<128, 1>::chunk(H, G) : Layout<64, 1>::chunk(H, G));
    return chunks * (long long)(wide ? Layout<128, 2>::chunk(H, G) : Layout<64, 2>::chunk(H, G));
}

// The gated delta rule: q and k of group g at columns q_col + g D and k_col + g D of the rows, v of head h at v_col + h DV; decay logits a
// ([N, H D], or [N, H] with per_head), update logits b [N, H]. scratch: llmie_chunk_scratch floats, 16-byte aligned.
LLMIE_API int llmie_chunk_delta(const bf16* qkv, int stride, int q_col, int k_col, int v_col, const bf16* a, int a_stride, const bf16* b, int b_stride,
                                const float* A_log, const float* dt_bias, float* scratch, float* state, const int* seq_starts, const int* seq_slots,
                                float* out, int H, int G, int D, int DV, int R, int max_len, float q_scale, float unit_eps, int per_head, cudaStream_t s) {
    if (!sizes_fit(H, G, D, DV, R, max_len) || ((uintptr_t)scratch & 15)) return LLMIE_ERR_BAD_ARGUMENT;
    const PrepareArgs pa{stride, q_col, k_col, a_stride, b_stride, A_log, dt_bias, seq_starts, scratch, H, G, D, q_scale, unit_eps};
    const ScanArgs<bf16> sa{scratch, qkv, stride, v_col, state, seq_starts, seq_slots, out, nullptr, H, G, D, DV};
    return per_head ? run_kind<KIND_DELTA_HEAD>(qkv, a, b, pa, sa, R, max_len, s) : run_kind<KIND_DELTA_CHANNEL>(qkv, a, b, pa, sa, R, max_len, s);
}

// The state-space recurrence: x of head h at x_col + h DV, B and C of group g at b_col + g NS and c_col + g NS of the rows; step sizes' logits dt.
LLMIE_API int llmie_chunk_ssm(const bf16* xbc, int stride, int x_col, int b_col, int c_col, const bf16* dt, int dt_stride, const float* A_log,
                              const float* dt_bias, const float* skip, float* scratch, float* state, const int* seq_starts, const int* seq_slots,
                              float* out, int H, int G, int NS, int DV, int R, int max_len, cudaStream_t s) {
    if (!sizes_fit(H, G, NS, DV, R, max_len) || ((uintptr_t)scratch & 15)) return LLMIE_ERR_BAD_ARGUMENT;
    const PrepareArgs pa{stride, c_col, b_col, dt_stride, 0, A_log, dt_bias, seq_starts, scratch, H, G, NS, 1.f, 0.f};
    const ScanArgs<bf16> sa{scratch, xbc, stride, x_col, state, seq_starts, seq_slots, out, skip, H, G, NS, DV};
    return run_kind<KIND_GIVEN>(xbc, dt, nullptr, pa, sa, R, max_len, s);
}
