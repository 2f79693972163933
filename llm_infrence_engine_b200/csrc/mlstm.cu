// The matrix memory with exponential gates (the mLSTM cell of xLSTM), as a recurrence over the rows of each request. T is the
// storage type of the projections (float or bfloat16); gates, their logarithms and exponentials, the running maximum, the memory
// and the normaliser are 32-bit.
//
// Per head, with q (already times dim^-1/2), k of D entries and v of DV, a log input gate i and a log forget gate f:
//   m_t = max(f_t + m_(t-1), i_t);  a_t = exp(f_t + m_(t-1) - m_t);  b_t = exp(i_t - m_t)
//   S_t = a_t S_(t-1) + b_t k_t v_t^T;   n_t = a_t n_(t-1) + b_t k_t;   o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
// S, n and m start at zero. The normaliser n is kept as one more column of the memory (a column whose v is 1), so a request's
// state is [H, DV + 1, D], column by column, plus m [H]. The scan leaves the numerators (S_t^T q_t and n_t . q_t) and m_t per
// token; the division, the norm of each head's result and the output gate are one kernel behind it.
//
// A step's batch is ragged (request r owns the rows seq_starts[r] .. seq_starts[r + 1] - 1, its state lives in row
// seq_slots[r]): a prompt portion of any length and a single decoded token are the same launch, a request's rows are walked in
// order, and the lanes that share a column depend on D alone, so a position's result does not depend on how the request was cut.
#include <math.h>

#include "common.cuh"
#include "scan_sums.cuh"

namespace {

constexpr int ML_THREADS = 128;
constexpr int ML_TILE = 16;   // tokens per stage, a token's gates per lane of the gates' warp
static inline __host__ __device__ constexpr int ml_parts(int dmax) { return dmax >= 32 ? dmax / 8 : 4; }

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
// ln sigmoid(x) = min(x, 0) - ln(1 + exp(-|x|))
__device__ __forceinline__ float log_sigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// One block per token: q (times q_scale) and k of every head as floats, and the two gates from their 32-bit pre-activations
// gates[n] = [W_i h (H) | W_f h (H)]:  i = cap tanh((x + b_i) / cap),  f = ln sigmoid(cap tanh((x + b_f) / cap)); cap <= 0: no cap.
template <typename T>
__global__ void __launch_bounds__(128) mlstm_prepare_kernel(const T* __restrict__ z, int z_stride, int q_col, int k_col, const float* __restrict__ gates,
                                                            int g_stride, const float* __restrict__ bias_i, const float* __restrict__ bias_f, float cap,
                                                            float q_scale, float* __restrict__ qf, float* __restrict__ kf, float* __restrict__ ig,
                                                            float* __restrict__ fg, int H, int D, const float* __restrict__ mstate, const int* __restrict__ seq_slots,
                                                            float* __restrict__ before, int R) {
    pdl_trigger();
    const int n = blockIdx.x;
    // the requests' m as the scan's blocks are to find it, whichever of them runs last: on its way while the block does its token (where the
    // requests' states lie was sent before the step's first kernel)
    const int mine = n * blockDim.x + threadIdx.x;
    const float* at = mine < R * H ? mstate + (size_t)seq_slots[mine / H] * H + mine % H : nullptr;
    pdl_wait();
    const float kept = at ? *at : 0.f;
    const T* row = z + (size_t)n * z_stride;
    const int HD = H * D;
    for (int i = threadIdx.x; i < HD; i += blockDim.x) {
        qf[(size_t)n * HD + i] = to_f32(row[q_col + i]) * q_scale;
        kf[(size_t)n * HD + i] = to_f32(row[k_col + i]);
    }
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        float xi = gates[(size_t)n * g_stride + h] + bias_i[h];
        float xf = gates[(size_t)n * g_stride + H + h] + bias_f[h];
        if (cap > 0.f) { xi = cap * tanhf(xi / cap); xf = cap * tanhf(xf / cap); }
        ig[(size_t)n * H + h] = xi;
        fg[(size_t)n * H + h] = log_sigmoid_f(xf);
    }
    if (at) before[mine] = kept;
    for (int i = mine + gridDim.x * blockDim.x; i < R * H; i += gridDim.x * blockDim.x) before[i] = mstate[(size_t)seq_slots[i / H] * H + i % H];
}

// Block (x, h, r): COLS columns of head h of request r, PARTS lanes (D / 8) to CPL columns side by side, each lane holding DPL entries of
// each in registers (16-byte pieces, PARTS pieces apart), in pairs for the packed multiply-add. Rows of q and k
// come in tiles of ML_TILE tokens through a two-stage ring (cp.async). A fifth warp does nothing but the gates: while the other four
// work on a tile it walks the chain of maxima over the next one and turns the gates into (a, b, m) per token, a token per lane, so the
// chain and the exponentials are nobody's wait. Nothing is reduced token by token: the lanes of a column add up PARTS sums together,
// each ending with one (parts_scatter). A full tile has no branch between its tokens, and a token's rows are loaded while the one
// before is worked on.
//
// The walk is bound by a token's instructions on one warp (its latency hides behind the next token's, nothing feeds back): with four
// columns to a group of 16 lanes on 80 blocks, a branch per token and the gates between two tiles on the first of the four warps, a
// prompt of 1,301 tokens (8 heads of 128 x 128, beside one of 700) took 659 us; this form 140 us.
//
// The request's m is read by every block of its (h, r) and written by one. They read it where the prepare kernel has put it (`before`), so that
// no block that starts late reads what an early one left.
template <typename T, int DMAX, int CPL>
__global__ void __launch_bounds__(ML_THREADS + 32) mlstm_scan_kernel(const T* __restrict__ v, int v_stride, int v_col, const float* __restrict__ qf,
                                                                     const float* __restrict__ kf, const float* __restrict__ ig, const float* __restrict__ fg,
                                                                     float* __restrict__ state, float* mstate, const int* __restrict__ seq_starts,
                                                                     const int* __restrict__ seq_slots, float* __restrict__ num, float* __restrict__ m_out,
                                                                     const float* __restrict__ before, int H, int D, int DV) {
    constexpr int PARTS = ml_parts(DMAX), DPL = DMAX / PARTS, COLS = ML_THREADS / PARTS * CPL, Q = DMAX / 4, P2 = DPL / 2, BATCH = PARTS / CPL;
    extern __shared__ __align__(16) float ml_smem[];
    float* k_s = ml_smem;                          // [2][ML_TILE][DMAX]
    float* q_s = k_s + 2 * ML_TILE * DMAX;
    float* v_s = q_s + 2 * ML_TILE * DMAX;         // [2][ML_TILE][COLS]
    float* a_s = v_s + 2 * ML_TILE * COLS;         // [2][ML_TILE]
    float* b_s = a_s + 2 * ML_TILE;
    pdl_wait();
    const int h = blockIdx.y, r = blockIdx.z;
    const int C = DV + 1;                 // the last column is the normaliser
    const int s0 = seq_starts[r], s1 = seq_starts[r + 1];
    const int slot = seq_slots[r];
    if (s1 - s0 < ML_TILE) pdl_trigger();   // (a short walk: the kernel behind may move in and set up)
    if (threadIdx.x >= ML_THREADS) {      // the warp of the gates
        const int lane = threadIdx.x - ML_THREADS;
        float m_carry = before[(size_t)r * H + h];
        float pre_i, pre_f;
        auto load = [&](int base) {
            pre_i = -INFINITY;
            pre_f = 0.f;
            if (lane < ML_TILE && base + lane < s1) {
                pre_i = ig[(size_t)(base + lane) * H + h];
                pre_f = fg[(size_t)(base + lane) * H + h];
            }
        };
        auto gates = [&](int base, int buf) {
            // the chain m -> max(f + m, i) over the tile's tokens, walked by every lane of the warp in the tokens' order (each step
            // exactly as a token-by-token walk would take it, so the bits do not depend on where a tile begins); lane t keeps token t's
            float m_run = m_carry, m_prev = m_carry, m_t = m_carry;
            const int count = min(ML_TILE, s1 - base);
            auto walk = [&](int t) {
                const float ft = __shfl_sync(0xffffffffu, pre_f, t), it = __shfl_sync(0xffffffffu, pre_i, t);
                const float m_new = fmaxf(ft + m_run, it);
                if (lane == t) { m_prev = m_run; m_t = m_new; }
                m_run = m_new;
            };
            // (decoded tokens: the other warps wait for this tile's gates, so the walk ends with the tokens there are. Short keys leave the chain the
            // longest part of a tile: there one run of instructions for both measured 8 to 11 % faster on prompts, longer keys two, by as much)
            if constexpr (DMAX <= 32) {
#pragma unroll
                for (int t = 0; t < ML_TILE; ++t)
                    if (t < count) walk(t);
            } else if (count == ML_TILE) {
#pragma unroll
                for (int t = 0; t < ML_TILE; ++t) walk(t);
            } else {
                for (int t = 0; t < count; ++t) walk(t);
            }
            if (lane < count) {
                a_s[buf * ML_TILE + lane] = expf(pre_f + m_prev - m_t);
                b_s[buf * ML_TILE + lane] = expf(pre_i - m_t);
                if (blockIdx.x == 0 && base + lane < s1) m_out[(size_t)(base + lane) * H + h] = m_t;
            }
            m_carry = m_run;
        };
        if (s0 < s1) {
            load(s0);
            gates(s0, 0);
            load(s0 + ML_TILE);
        }
        int buf = 0;
        for (int base = s0; base < s1; base += ML_TILE, buf ^= 1) {
            __syncthreads();
            if (base + ML_TILE < s1) {
                gates(base + ML_TILE, buf ^ 1);
                load(base + 2 * ML_TILE);
            }
        }
        pdl_trigger();
        if (blockIdx.x == 0 && lane == 0 && s0 < s1) mstate[(size_t)slot * H + h] = m_carry;
        return;
    }
    const int part = threadIdx.x % PARTS, my_col = threadIdx.x / PARTS * CPL;   // the first of the lane's CPL columns, within the block
    const int col = blockIdx.x * COLS + my_col;
    const bool vec = (D & 3) == 0, vec_state = vec && ((uintptr_t)state & 15) == 0;
    float* st = state + ((size_t)slot * H + h) * C * D;
    float2 S[CPL][P2];
#pragma unroll
    for (int u = 0; u < CPL; ++u)
#pragma unroll
        for (int i = 0; i < DPL / 4; ++i) {
            const int d = 4 * PARTS * i + 4 * part;
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (DMAX != 128 && vec_state) {   // (16 bytes at a time the walk of 128 entries comes out 14 % slower on a prompt, 219 -> 252 us at 2,048 tokens)
                if (col + u < C && d < D) load4(st + (size_t)(col + u) * D + d, x);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (col + u < C && d + c < D) x[c] = st[(size_t)(col + u) * D + d + c];
            }
            S[u][2 * i] = make_float2(x[0], x[1]);
            S[u][2 * i + 1] = make_float2(x[2], x[3]);
        }
    auto fetch = [&](int base, int buf) {
        const int count = min(ML_TILE, s1 - base);
        for (int i = threadIdx.x; i < count * Q; i += ML_THREADS) {
            const int t = i / Q, d = (i % Q) * 4;
            const size_t off = ((size_t)(base + t) * H + h) * D + d;
            float *kd = k_s + (buf * ML_TILE + t) * DMAX + d, *qd = q_s + (buf * ML_TILE + t) * DMAX + d;
            if (vec && d < D) {
                cp_async16(kd, kf + off);
                cp_async16(qd, qf + off);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    kd[c] = d + c < D ? kf[off + c] : 0.f;
                    qd[c] = d + c < D ? qf[off + c] : 0.f;
                }
            }
        }
    };
    // the block's columns of v, into registers a tile ahead
    constexpr int VPT = (ML_TILE * COLS + ML_THREADS - 1) / ML_THREADS;
    T pre_v[VPT];   // (as they are stored: converted here, they would be waited for here)
    auto load_v = [&](int base) {
        const int count = min(ML_TILE, s1 - base);
#pragma unroll
        for (int n = 0; n < VPT; ++n) {
            const int j = threadIdx.x + n * ML_THREADS;
            const int t = j / COLS, c = blockIdx.x * COLS + j % COLS;
            pre_v[n] = from_f32<T>(c == DV ? 1.f : 0.f);
            if (j < count * COLS && c < DV) pre_v[n] = v[(size_t)(base + t) * v_stride + v_col + h * DV + c];
        }
    };
    auto store_v = [&](int buf) {
#pragma unroll
        for (int n = 0; n < VPT; ++n) {
            const int j = threadIdx.x + n * ML_THREADS;
            if (j < ML_TILE * COLS) v_s[buf * ML_TILE * COLS + j] = to_f32(pre_v[n]);
        }
    };
    if (s0 < s1) {
        fetch(s0, 0);
        load_v(s0);
    }
    cp_commit();
    int buf = 0;
    for (int base = s0; base < s1; base += ML_TILE, buf ^= 1) {
        const int count = min(ML_TILE, s1 - base);
        store_v(buf);                          // (this stage's last readers passed the barrier of the tile between)
        cp_wait<0>();
        __syncthreads();                       // this tile is in shared memory, and everyone is done with the other stage
        if (base + ML_TILE < s1) {
            fetch(base + ML_TILE, buf ^ 1);
            load_v(base + ML_TILE);
        }
        cp_commit();
        const float* kb = k_s + buf * ML_TILE * DMAX + 4 * part;
        const float* qb = q_s + buf * ML_TILE * DMAX + 4 * part;
        struct Row { float2 k[P2], q[P2]; };
        auto load_row = [&](int t, Row& w) {
#pragma unroll
            for (int i = 0; i < DPL / 4; ++i) {
                const float4 k4 = *reinterpret_cast<const float4*>(kb + t * DMAX + 4 * PARTS * i);
                const float4 q4 = *reinterpret_cast<const float4*>(qb + t * DMAX + 4 * PARTS * i);
                w.k[2 * i] = make_float2(k4.x, k4.y); w.k[2 * i + 1] = make_float2(k4.z, k4.w);
                w.q[2 * i] = make_float2(q4.x, q4.y); w.q[2 * i + 1] = make_float2(q4.z, q4.w);
            }
        };
        auto token = [&](int t, const Row& w, float* y) {   // y[u]: this lane's share of S^T q of its columns
            const float a = a_s[buf * ML_TILE + t], b = b_s[buf * ML_TILE + t];
            const float2 a2 = make_float2(a, a);
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                const float bv = b * v_s[(buf * ML_TILE + t) * COLS + my_col + u];
                const float2 bv2 = make_float2(bv, bv);
                float2 sum[2];
                sum[0] = sum[1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < P2; ++i) {
                    S[u][i] = fma2(bv2, w.k[i], mul2(a2, S[u][i]));
                    sum[i & 1] = fma2(S[u][i], w.q[i], sum[i & 1]);
                }
                y[u] = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            }
        };
        float* o = num + ((size_t)base * H + h) * C + col;
        if (count == ML_TILE) {
            const int my_t = part / CPL, my_u = part % CPL;   // the sum of a batch that this lane ends with
            Row now;
            load_row(0, now);
#pragma unroll
            for (int t0 = 0; t0 < ML_TILE; t0 += BATCH) {
                float y[PARTS];
#pragma unroll
                for (int t = 0; t < BATCH; ++t) {
                    Row next;
                    if (t0 + t + 1 < ML_TILE) load_row(t0 + t + 1, next);
                    token(t0 + t, now, y + t * CPL);
                    now = next;
                }
                const float mine = parts_scatter<PARTS>(y, part);
                if (col + my_u < C) o[(size_t)(t0 + my_t) * H * C + my_u] = mine;
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
                    if (col + u < C && part == 0) o[(size_t)t * H * C + u] = sum;
                }
            }
        }
    }
    cp_wait<0>();
    pdl_trigger();
#pragma unroll
    for (int u = 0; u < CPL; ++u)
#pragma unroll
        for (int i = 0; i < DPL / 4; ++i) {
            const int d = 4 * PARTS * i + 4 * part;
            const float x[4] = {S[u][2 * i].x, S[u][2 * i].y, S[u][2 * i + 1].x, S[u][2 * i + 1].y};
            if (vec_state) {
                if (col + u < C && d < D) store4(st + (size_t)(col + u) * D + d, x);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (col + u < C && d + c < D) st[(size_t)(col + u) * D + d + c] = x[c];
            }
        }
}

// One block per (token, head): o = num / (max(|n . q|, exp(-m)) + 1e-6); o / sqrt(mean(o^2) + eps) * w[h * DV + j] * sigmoid(gate).
template <typename T>
__global__ void __launch_bounds__(128) mlstm_finish_kernel(const float* __restrict__ num, const float* __restrict__ m_t, const T* __restrict__ gate,
                                                           int gate_stride, const float* __restrict__ w, T* __restrict__ out, int H, int DV, float eps) {
    __shared__ float scratch[36];
    pdl_trigger();
    pdl_wait();
    const int n = blockIdx.x, h = blockIdx.y;
    const float* row = num + ((size_t)n * H + h) * (DV + 1);
    const float den = fmaxf(fabsf(row[DV]), expf(-m_t[(size_t)n * H + h])) + 1e-6f;
    float sq = 0.f;
    for (int j = threadIdx.x; j < DV; j += blockDim.x) { const float o = row[j] / den; sq = fmaf(o, o, sq); }
    const float rstd = 1.0f / sqrtf(block_sum(sq, scratch) / (float)DV + eps);
    for (int j = threadIdx.x; j < DV; j += blockDim.x) {
        const float o = row[j] / den;
        const float g = sigmoid_f(to_f32(gate[(size_t)n * gate_stride + (size_t)h * DV + j]));
        out[((size_t)n * H + h) * DV + j] = from_f32<T>(o * rstd * w[(size_t)h * DV + j] * g);
    }
}

template <typename T, int DM, int CPL>
int launch_scan_as(const T* v, int v_stride, int v_col, const float* qf, const float* kf, const float* ig, const float* fg, float* state, float* mstate,
                   const int* seq_starts, const int* seq_slots, float* num, float* m_out, const float* before, int H, int D, int DV, int R, bool alone,
                   cudaStream_t s) {
    constexpr int COLS = ML_THREADS / ml_parts(DM) * CPL;
    constexpr int smem = 4 * 2 * ML_TILE * (2 * DM + COLS + 2);
    if (smem > 48 * 1024) {
        static OncePerDevice granted;
        if (const int rc = grant_shared(granted, mlstm_scan_kernel<T, DM, CPL>, smem)) return rc;
    }
    const dim3 grid((DV + 1 + COLS - 1) / COLS, H, R);
    return launch_kernel_on(alone, mlstm_scan_kernel<T, DM, CPL>, grid, dim3(ML_THREADS + 32), (size_t)smem, s, v, v_stride, v_col, qf, kf, ig, fg, state,
                            mstate, seq_starts, seq_slots, num, m_out, before, H, D, DV);
}

// The lanes that share a column depend on the padded key size alone, never on the batch: the order of every sum, and with it every bit. How
// many columns a lane has changes no sum: four where the step's columns are more than fill the device two at a time.
template <typename T>
int launch_scan(const T* v, int v_stride, int v_col, const float* qf, const float* kf, const float* ig, const float* fg, float* state, float* mstate,
                const int* seq_starts, const int* seq_slots, float* num, float* m_out, const float* before, int H, int D, int DV, int R, bool alone,
                cudaStream_t s) {
#define ML_ARGS v, v_stride, v_col, qf, kf, ig, fg, state, mstate, seq_starts, seq_slots, num, m_out, before, H, D, DV, R, alone, s
    const long long columns = (long long)R * H * (DV + 1);
#define ML_AS(DM) return columns * ml_parts(DM) > 148LL * ML_THREADS * 2 ? launch_scan_as<T, DM, 4>(ML_ARGS) : launch_scan_as<T, DM, 2>(ML_ARGS)
    if (D <= 16) ML_AS(16);
    if (D <= 32) ML_AS(32);
    if (D <= 64) ML_AS(64);
    if (D <= 128) ML_AS(128);
    ML_AS(256);
#undef ML_AS
#undef ML_ARGS
}

}  // namespace

// z [N, z_stride] holds q (H * D from q_col) and k (from k_col); gates [N, g_stride] float = [W_i h | W_f h]; outputs qf, kf [N, H, D],
// ig, fg [N, H], all float; before [R, H]: the m of each of the step's requests (mstate [slots, H]).
LLMIE_API int llmie_mlstm_prepare(const void* z, int z_stride, int q_col, int k_col, const float* gates, int g_stride, const float* bias_i,
                                  const float* bias_f, float cap, float q_scale, float* qf, float* kf, float* ig, float* fg, const float* mstate,
                                  const int* seq_slots, float* before, int R,
                                  int N, int H, int D, int dtype, cudaStream_t s) {
    if (N <= 0) return 0;
    if (H <= 0 || D <= 0 || g_stride < 2 * H || q_col < 0 || k_col < 0 || !bias_i || !bias_f || !mstate || !seq_slots || !before || R < 0) return LLMIE_ERR_BAD_ARGUMENT;
    if (dtype == DT_F32)
        return launch_kernel(mlstm_prepare_kernel<float>, dim3(N), dim3(128), 0, s, (const float*)z, z_stride, q_col, k_col, gates, g_stride, bias_i, bias_f,
                             cap, q_scale, qf, kf, ig, fg, H, D, mstate, seq_slots, before, R);
    return launch_kernel(mlstm_prepare_kernel<bf16>, dim3(N), dim3(128), 0, s, (const bf16*)z, z_stride, q_col, k_col, gates, g_stride, bias_i, bias_f, cap,
                         q_scale, qf, kf, ig, fg, H, D, mstate, seq_slots, before, R);
}

// v: DV columns per head from v_col of rows of v_stride; state [slots, H, DV + 1, D], mstate [slots, H]; num [N, H, DV + 1], m_out [N, H]; before [R, H]: from the prepare kernel.
LLMIE_API int llmie_mlstm_scan(const void* v, int v_stride, int v_col, const float* qf, const float* kf, const float* ig, const float* fg, float* state,
                               float* mstate, const int* seq_starts, const int* seq_slots, float* num, float* m_out, const float* before, int H, int D, int DV, int R,
                               int max_rows, int dtype, cudaStream_t s) {
    if (R <= 0) return 0;
    if (H <= 0 || H > 65535 || R > 65535 || D <= 0 || D > 256 || DV <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    const bool alone = max_rows >= 64;   // a long walk: see launch_kernel_on
    if (dtype == DT_F32) return launch_scan<float>((const float*)v, v_stride, v_col, qf, kf, ig, fg, state, mstate, seq_starts, seq_slots, num, m_out, before, H, D, DV, R, alone, s);
    return launch_scan<bf16>((const bf16*)v, v_stride, v_col, qf, kf, ig, fg, state, mstate, seq_starts, seq_slots, num, m_out, before, H, D, DV, R, alone, s);
}

// gate: H * DV columns of rows of gate_stride (storage type); w [H * DV]; out [N, H * DV] of the storage type.
LLMIE_API int llmie_mlstm_finish(const float* num, const float* m_t, const void* gate, int gate_stride, const float* w, void* out, int N, int H, int DV,
                                 float eps, int dtype, cudaStream_t s) {
    if (N <= 0) return 0;
    if (H <= 0 || H > 65535 || DV <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    int threads = 32;
    while (threads < 128 && threads < DV) threads *= 2;
    if (dtype == DT_F32)
        return launch_kernel(mlstm_finish_kernel<float>, dim3(N, H), dim3(threads), 0, s, num, m_t, (const float*)gate, gate_stride, w, (float*)out, H, DV, eps);
    return launch_kernel(mlstm_finish_kernel<bf16>, dim3(N, H), dim3(threads), 0, s, num, m_t, (const bf16*)gate, gate_stride, w, (bf16*)out, H, DV, eps);
}
