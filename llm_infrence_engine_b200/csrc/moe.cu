// A feed-forward of routed experts: the router's choice, the tokens sorted by expert, the experts' two products over the sorted
// rows (a grouped product: every tile of rows belongs to one expert and multiplies by that expert's matrix), and the weighted sum
// back into the residual stream. Everything is decided on the device (no host read of a count), so a step with routed experts is
// captured in a CUDA graph like any other. T is the storage type of activations and matrices (float or bfloat16); router scores,
// weights and the sum into the stream are 32-bit.
//
// The result of a token does not depend on what else is in the batch: a row of a grouped product is a sum over K in one fixed
// order whatever tile it falls into, and the weighted sum adds a token's experts in the order of its choice.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int ROUTE_MAX_PER_LANE = 16;   // up to 512 router outputs
constexpr int MOE_TM = 4;                // most rows of a tile of the grouped product on the CUDA cores
constexpr int MOE_COLS = 32;             // outputs per block there
constexpr int MOE_ROWS_SMEM = 96 * 1024; // what a tile's rows may take of shared memory
constexpr int SORT_THREADS = 1024;
constexpr int SORT_MAX_EXPERTS = 4096;

// One warp per token: s = softmax(logits) over all `total` router outputs; the `top` outputs with the largest s + correction are
// chosen (of equal scores the lower index first); their weights are s / (sum of the chosen s + 1e-20).
// (one warp: token n's row of logits, in global or shared memory)
// `scoring` 1 instead: s = sigmoid(logits), every output by itself, and the weights are the chosen s as they are (not renormalised).
// `scoring` 2: the `top` largest logits are chosen, and their weights are the softmax over the chosen ones alone.
// `bias` [total] or null is added to the logits first.
template <int PER_LANE>
__device__ __forceinline__ void route_token_as(const float* __restrict__ row, const float* __restrict__ correction, int* __restrict__ ids,
                                               float* __restrict__ weights, int n, int total, int top, int lane, int scoring,
                                               const float* __restrict__ bias) {
    float s[PER_LANE], c[PER_LANE];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int e = lane + 32 * j;
        s[j] = e < total ? row[e] + (bias ? bias[e] : 0.f) : -INFINITY;
        c[j] = s[j];
        mx = fmaxf(mx, s[j]);
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int e = lane + 32 * j;
        if (scoring == 1) s[j] = e < total ? 1.0f / (1.0f + expf(-s[j])) : 0.f;
        else s[j] = e < total ? expf(s[j] - mx) : 0.f;
        sum += s[j];
    }
    sum = scoring != 0 ? 1.f : warp_sum(sum);
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int e = lane + 32 * j;
        s[j] = s[j] / sum;
        if (scoring != 2) c[j] = e < total ? s[j] + (correction ? correction[e] : 0.f) : -INFINITY;
    }
    float chosen_sum = 0.f;
    float my_w = 0.f;      // lane k keeps the k-th choice
    int my_id = 0;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {
            const int e = lane + 32 * j;
            if (c[j] > best) { best = c[j]; best_e = e; }   // (ascending e within a lane: the lower index wins a tie)
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
        }
        float w = 0.f;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j)
            if (lane + 32 * j == best_e) { w = s[j]; c[j] = -INFINITY; }
        w = warp_sum(w);   // only the owner's lane holds it
        chosen_sum += w;
        if (lane == (k & 31)) { my_w = w; my_id = best_e; }
        if ((k & 31) == 31 || k == top - 1) {   // (more than 32 choices: written in rounds)
            // weights are divided below, once the sum is known: keep raw values in global memory for now
            const int k0 = k & ~31;
            if (k0 + lane <= k) { ids[(size_t)n * top + k0 + lane] = my_id; weights[(size_t)n * top + k0 + lane] = my_w; }
        }
    }
    __syncwarp();
    const float inv = scoring == 1 ? 1.0f : 1.0f / (chosen_sum + (scoring == 0 ? 1e-20f : 0.f));   // (2: the largest logit's share is 1)
    for (int k = lane; k < top; k += 32) weights[(size_t)n * top + k] *= inv;
}
// (a lane's share of the outputs as a compile-time number: with room for 512 outputs, 16 of them spend sixteen times the instructions)
static inline __host__ __device__ int route_per_lane(int total) { return total <= 32 ? 1 : (total <= 128 ? 4 : ROUTE_MAX_PER_LANE); }
__device__ __forceinline__ void route_token(const float* __restrict__ row, const float* __restrict__ correction, int* __restrict__ ids,
                                            float* __restrict__ weights, int n, int total, int top, int lane, int scoring,
                                            const float* __restrict__ bias) {
    const int per_lane = route_per_lane(total);
    if (per_lane == 1) route_token_as<1>(row, correction, ids, weights, n, total, top, lane, scoring, bias);
    else if (per_lane == 4) route_token_as<4>(row, correction, ids, weights, n, total, top, lane, scoring, bias);
    else route_token_as<ROUTE_MAX_PER_LANE>(row, correction, ids, weights, n, total, top, lane, scoring, bias);
}

// Rows of `total + extra` logits; the extra ones are gates of their own: gates[n][j] = sigmoid(logit).
template <int PER_LANE>
__global__ void __launch_bounds__(128) moe_route_kernel(const float* __restrict__ logits, const float* __restrict__ correction,
                                                        int* __restrict__ ids, float* __restrict__ weights, int N, int total, int top, int scoring,
                                                        const float* __restrict__ bias, int extra, float* __restrict__ gates) {
    pdl_trigger();
    pdl_wait();
    const int n = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (n >= N) return;
    const float* row = logits + (size_t)n * (total + extra);
    const int lane = threadIdx.x & 31;
    for (int j = lane; j < extra; j += 32) gates[(size_t)n * extra + j] = 1.0f / (1.0f + expf(-row[total + j]));
    route_token_as<PER_LANE>(row, correction, ids, weights, n, total, top, lane, scoring, bias);
}

// The router's product and its choice in one kernel, a block per token: the token's row lies in shared memory as floats, the warps
// share the router's outputs (a warp's lanes walk an output's weight row in 16-byte pieces; the sum runs over K in one order whatever
// the step holds), and the first warp chooses from the logits in shared memory. For the few rows of a decode step, where the product
// alone would be a kernel that walks K in one block. EARLY: no warp has more than ROUTER_EARLY pieces of the matrix, and (at rest) they are
// all asked for before the kernel ahead has finished. More pieces that many at a time cost more in counting than they save (64 outputs of 1,024
// in float32: output by output 7.0 us, in four rounds of pieces 9.6), and with more blocks than multiprocessors eight warps each do better than
// sixteen. (8 rows, K = 1,024, 18 outputs, float32: 10.5 us with eight warps and the choice's room for 512 outputs, 4.1 now.)
constexpr int ROUTER_THREADS = 512;
constexpr int ROUTER_EARLY = 8;
template <typename T, bool EARLY>
__global__ void __launch_bounds__(ROUTER_THREADS) moe_router_kernel(const T* __restrict__ h, const T* __restrict__ w, const float* __restrict__ correction,
                                                                    int* __restrict__ ids, float* __restrict__ weights, int K, int total, int top, int scoring,
                                                                    const float* __restrict__ bias, int extra, float* __restrict__ gates, int at_rest) {
    extern __shared__ __align__(16) float router_smem[];   // [K] the row, then [total + extra] the logits
    constexpr int VN = Vec16<T>::N;
    float* row = router_smem;
    float* logits = router_smem + ((K + 3) & ~3);
    pdl_trigger();
    const int n = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = (K % VN) == 0 && ((uintptr_t)h & 15) == 0 && ((uintptr_t)w & 15) == 0;
    // a warp's pieces of the matrix: outputs warp, warp + warps, ..., each in steps of 32 * VN entries
    const int warps = blockDim.x >> 5, steps = (K + 32 * VN - 1) / (32 * VN), outputs = total + extra;
    uint4 early[ROUTER_EARLY];
    if constexpr (EARLY) {
        pdl_wait_unless(at_rest);
        int e = warp, step = 0;   // (counted on: a division per piece costs more than its multiply-adds)
#pragma unroll
        for (int i = 0; i < ROUTER_EARLY; ++i) {
            const int k = (step * 32 + lane) * VN;
            early[i] = make_uint4(0u, 0u, 0u, 0u);
            if (e < outputs && k < K) early[i] = *reinterpret_cast<const uint4*>(w + (size_t)e * K + k);
            if (++step == steps) { step = 0; e += warps; }
        }
    }
    pdl_wait();
    const T* src = h + (size_t)n * K;
    if (vec) {
        for (int k = threadIdx.x * VN; k < K; k += blockDim.x * VN) {
            float v[VN];
            Vec16<T>::load(src + k, v);
#pragma unroll
            for (int i = 0; i < VN; ++i) row[k + i] = v[i];
        }
    } else {
        for (int k = threadIdx.x; k < K; k += blockDim.x) row[k] = to_f32(src[k]);
    }
    __syncthreads();
    if constexpr (EARLY) {
        float acc = 0.f;
        int e = warp, step = 0;
#pragma unroll
        for (int i = 0; i < ROUTER_EARLY; ++i) {
            if (e < outputs) {
                const int k = (step * 32 + lane) * VN;
                if (k < K) {
                    float v[VN];
                    Vec16<T>::load(reinterpret_cast<const T*>(&early[i]), v);
#pragma unroll
                    for (int c = 0; c < VN; ++c) acc = fmaf(row[k + c], v[c], acc);
                }
                if (++step == steps) {
                    acc = warp_sum(acc);
                    if (lane == 0) logits[e] = acc;
                    acc = 0.f;
                    step = 0;
                    e += warps;
                }
            }
        }
    } else {
        for (int e = warp; e < outputs; e += warps) {
            const T* we = w + (size_t)e * K;
            float acc = 0.f;
            if (vec) {
                for (int k = lane * VN; k < K; k += 32 * VN) {
                    float v[VN];
                    Vec16<T>::load(we + k, v);
#pragma unroll
                    for (int i = 0; i < VN; ++i) acc = fmaf(row[k + i], v[i], acc);
                }
            } else {
                for (int k = lane; k < K; k += 32) acc = fmaf(row[k], to_f32(we[k]), acc);
            }
            acc = warp_sum(acc);
            if (lane == 0) logits[e] = acc;
        }
    }
    __syncthreads();
    if (warp == 1)
        for (int j = lane; j < extra; j += 32) gates[(size_t)n * extra + j] = 1.0f / (1.0f + expf(-logits[total + j]));
    if (warp == 0) route_token(logits, correction, ids, weights, n, total, top, lane, scoring, bias);
}

// (The experts laid out by one thread one after the other, and 1,024 threads for a decode step's few pairs: 3.4 to 3.7 us, 1.8 to 2.3 here.)
// One block: the step's (token, choice) pairs counted per expert, the experts' runs laid out one behind the other, every pair
// given a place in its expert's run, and the runs cut into tiles of `tile_rows` rows. Choices of identity experts (ids >= E)
// take no place (place_of = -1).
//   offsets [E + 1]; perm [pairs]: place -> pair; place_of [pairs]: pair -> place or -1;
//   tiles [1 + 2 * max_tiles]: the number of tiles, then (expert, first place) of each
__global__ void __launch_bounds__(SORT_THREADS) moe_sort_kernel(const int* __restrict__ ids, int pairs, int E, int tile_rows, int* __restrict__ offsets,
                                                                 int* __restrict__ perm, int* __restrict__ place_of, int* __restrict__ tiles, int max_tiles) {
    __shared__ int count[SORT_MAX_EXPERTS];
    __shared__ int cursor[SORT_MAX_EXPERTS];
    pdl_trigger();
    for (int e = threadIdx.x; e < E; e += blockDim.x) count[e] = 0;
    pdl_wait();
    __syncthreads();
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int e = ids[i];
        if (e >= 0 && e < E) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // an expert per lane, 32 at a time: where its run and its tiles begin
        int at = 0, nt = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + threadIdx.x, mine = e < E ? count[e] : 0, my_tiles = (mine + tile_rows - 1) / tile_rows;
            int rows = mine, upto = my_tiles;   // of the experts up to this lane's
#pragma unroll
            for (int o = 1; o < 32; o *= 2) {
                const int r = __shfl_up_sync(0xffffffffu, rows, o), u = __shfl_up_sync(0xffffffffu, upto, o);
                if ((int)threadIdx.x >= o) { rows += r; upto += u; }
            }
            const int first = at + rows - mine, tile = nt + upto - my_tiles;
            if (e < E) {
                offsets[e] = first;
                cursor[e] = first;
                for (int k = 0; k < my_tiles && tile + k < max_tiles; ++k) { tiles[1 + 2 * (tile + k)] = e; tiles[2 + 2 * (tile + k)] = first + k * tile_rows; }
            }
            at += __shfl_sync(0xffffffffu, rows, 31);
            nt += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (threadIdx.x == 0) {
            offsets[E] = at;
            tiles[0] = min(nt, max_tiles);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int e = ids[i];
        if (e >= 0 && e < E) {
            const int p = atomicAdd(&cursor[e], 1);
            perm[p] = i;
            place_of[i] = p;
        } else {
            place_of[i] = -1;
        }
    }
}

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

// The grouped product on the CUDA cores for FEW rows per expert (decode steps) and for float32: a tile is up to `tile_rows` (at
// most MOE_TM) places of one expert, whose rows of K numbers lie in shared memory as floats; a block owns MOE_COLS outputs, a warp
// MOE_COLS / 8 of them, taken together: the lanes walk the outputs' weight rows (and, GATED, the up rows of the same outputs)
// 16 bytes at a time, so the matrices are read once per tile in full lines, which is what bounds a decode step.
//   GATED: out[place, j] = silu(a . Wg[e][j]) * (a . Wu[e][j]) with W [E][2 F][K] (an expert's gate rows, then its up rows), out of type TO;
//          with limit > 0 the unit is min(g, limit) * sigmoid(alpha g) * (clamp(u, -limit, limit) + shift);
//          with row_scale the row a is first multiplied by row_scale[pair] (a weight on the expert's input, rounded as it would be stored)
//   else:  out[place, j] = a . W[e][j] with W [E][F][K]
// The row a of a place is x[row_map[place] / row_div] (the token of the pair that sits there), or x[place] without a map.
// A sum runs over K in one order whatever the tile holds: a place's result does not depend on its neighbours.
template <typename T, typename TO, bool GATED>
__global__ void __launch_bounds__(256, 2) moe_rows_kernel(const T* __restrict__ x, const int* __restrict__ row_map, int row_div, const T* __restrict__ w,
                                                       const int* __restrict__ offsets, const int* __restrict__ tiles, TO* __restrict__ out, int F,
                                                       int K, int tile_rows, const float* __restrict__ row_scale, float limit, float alpha, float shift) {
    extern __shared__ __align__(16) float moe_rows_smem[];   // [tile_rows][K]
    constexpr int VN = Vec16<T>::N;
    pdl_trigger();
    pdl_wait();
    if ((int)blockIdx.y >= tiles[0]) return;
    const int e = tiles[1 + 2 * blockIdx.y], p0 = tiles[2 + 2 * blockIdx.y];
    const int count = min(offsets[e + 1] - p0, tile_rows);
    const bool vec = (K % VN) == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* we = w + (size_t)e * (GATED ? 2 : 1) * F * K;
    constexpr int CPW = MOE_COLS / 8;   // a warp's outputs, taken together: their weight rows are in flight at once
    const int j0 = blockIdx.x * MOE_COLS + warp * CPW;
    const T* wrow[CPW];
#pragma unroll
    for (int c = 0; c < CPW; ++c) wrow[c] = we + (size_t)min(j0 + c, F - 1) * K;   // (an output past the end repeats the last: not stored)
    const size_t up = (size_t)F * K;   // from an output's gate row to its up row (read only when GATED)
    // a step's 16-byte pieces of all the warp's weight rows. GATED in bfloat16: the next step's are asked for before this one's are used, the
    // first step's before the tile's rows are fetched (2 rows, 16 experts of 512 x 1,024: 8.5 -> 7.8 us, 8 rows: equal; without a gate, with half the
    // pieces, the registers cost more than it gains: 7.0 -> 7.6 at 8 rows; so they do in float32: both products 24.2 -> 25.2 at 16 rows of 512, 8 experts)
    constexpr bool AHEAD = GATED && sizeof(T) == 2;
    struct Pieces { uint4 g[CPW], u[GATED ? CPW : 1]; };
    auto ask = [&](int k, Pieces& p) {
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
            p.g[c] = *reinterpret_cast<const uint4*>(wrow[c] + k);
            if constexpr (GATED) p.u[c] = *reinterpret_cast<const uint4*>(wrow[c] + up + k);
        }
    };
    Pieces now;
    if (AHEAD && vec && lane * VN < K) ask(lane * VN, now);
    for (int r = 0; r < count; ++r) {
        const int p = p0 + r;
        const T* src = x + (size_t)(row_map ? row_map[p] / row_div : p) * K;
        const float rs = (row_scale && row_map) ? row_scale[row_map[p]] : 1.f;   // the pair's weight on the expert's INPUT
        float* dst = moe_rows_smem + (size_t)r * K;
        if (vec) {
            for (int k = threadIdx.x * VN; k < K; k += 256 * VN) {
                float v[VN];
                Vec16<T>::load(src + k, v);
#pragma unroll
                for (int i = 0; i < VN; ++i) dst[k + i] = row_scale ? round_through<T>(v[i] * rs) : v[i];
            }
        } else {
            for (int k = threadIdx.x; k < K; k += 256) dst[k] = row_scale ? round_through<T>(to_f32(src[k]) * rs) : to_f32(src[k]);
        }
    }
    __syncthreads();
    if (j0 >= F) return;
    float ag[CPW][MOE_TM] = {}, au[GATED ? CPW : 1][MOE_TM] = {};
    if (vec) {
        for (int k = lane * VN; k < K; k += 32 * VN) {
            Pieces next;
            if constexpr (!AHEAD) ask(k, now);
            else if (k + 32 * VN < K) ask(k + 32 * VN, next);
#pragma unroll
            for (int i = 0; i < VN; i += 4) {   // (four entries of every piece at a time as floats: all of them would not fit the registers)
                float g[CPW][4], u[GATED ? CPW : 1][4];
#pragma unroll
                for (int c = 0; c < CPW; ++c) {
                    load4(reinterpret_cast<const T*>(&now.g[c]) + i, g[c]);
                    if constexpr (GATED) load4(reinterpret_cast<const T*>(&now.u[c]) + i, u[c]);
                }
#pragma unroll
                for (int r = 0; r < MOE_TM; ++r) {
                    if (r < count) {
                        const float4 av = *reinterpret_cast<const float4*>(moe_rows_smem + (size_t)r * K + k + i);
#pragma unroll
                        for (int c = 0; c < CPW; ++c) {
                            ag[c][r] = fmaf(av.x, g[c][0], ag[c][r]); ag[c][r] = fmaf(av.y, g[c][1], ag[c][r]);
                            ag[c][r] = fmaf(av.z, g[c][2], ag[c][r]); ag[c][r] = fmaf(av.w, g[c][3], ag[c][r]);
                            if constexpr (GATED) {
                                float& s = au[c][r];
                                s = fmaf(av.x, u[c][0], s); s = fmaf(av.y, u[c][1], s);
                                s = fmaf(av.z, u[c][2], s); s = fmaf(av.w, u[c][3], s);
                            }
                        }
                    }
                }
            }
            if constexpr (AHEAD) now = next;
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            float g[CPW], u[GATED ? CPW : 1];
#pragma unroll
            for (int c = 0; c < CPW; ++c) {
                g[c] = to_f32(wrow[c][k]);
                if (GATED) u[GATED ? c : 0] = to_f32(wrow[c][up + k]);
            }
#pragma unroll
            for (int r = 0; r < MOE_TM; ++r) {
                if (r < count) {
                    const float a = moe_rows_smem[(size_t)r * K + k];
#pragma unroll
                    for (int c = 0; c < CPW; ++c) {
                        ag[c][r] = fmaf(a, g[c], ag[c][r]);
                        if (GATED) au[GATED ? c : 0][r] = fmaf(a, u[GATED ? c : 0], au[GATED ? c : 0][r]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < MOE_TM; ++r) {
        if (r < count) {
#pragma unroll
            for (int c = 0; c < CPW; ++c) {
                const float sg = warp_sum(ag[c][r]);
                const float su = GATED ? warp_sum(au[GATED ? c : 0][r]) : 0.f;
                float res = sg;
                if (GATED) {
                    if (limit > 0.f) {   // the clamped unit
                        const float g = fminf(sg, limit), u = fminf(fmaxf(su, -limit), limit) + shift;
                        res = g / (1.0f + expf(-alpha * g)) * u;
                    } else {
                        res = silu_f(sg) * su;
                    }
                }
                if (lane == 0 && j0 + c < F) out[(size_t)(p0 + r) * F + j0 + c] = from_f32<TO>(res);
            }
        }
    }
}

// xs[place] = x[perm[place] / top] (times row_scale[perm[place]], where given) for the places that the sort filled (offsets[E] of them): the rows of the tokens, in the order
// of their experts, as the tensor-core grouped product reads them. One block per place.
__global__ void moe_gather_kernel(const bf16* __restrict__ x, const int* __restrict__ perm, const int* __restrict__ offsets, int E, int top,
                                  bf16* __restrict__ xs, int K, const float* __restrict__ row_scale) {
    pdl_trigger();
    pdl_wait();
    const int p = blockIdx.x;
    if (p >= offsets[E]) return;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(perm[p] / top) * K);
    uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)p * K);
    if (!row_scale) {
        for (int i = threadIdx.x; i < K / 8; i += blockDim.x) dst[i] = src[i];
        return;
    }
    const float rs = row_scale[perm[p]];   // the pair's weight on the expert's input
    for (int i = threadIdx.x; i < K / 8; i += blockDim.x) {
        float v[8];
        Vec16<bf16>::load(reinterpret_cast<const bf16*>(src + i), v);
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j] * rs, v[2 * j + 1] * rs);
            w[j] = *reinterpret_cast<const uint32_t*>(&b);
        }
        dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// residual[t] += sum_k weight[t, k] * (y[place_of[t, k]] for an expert with matrices, h[t] itself for an identity expert), the
// experts of a token in the order of its choice. Block (t, c): COMBINE_VEC columns per thread of token t from column
// c * blockDim.x * COMBINE_VEC on; the rows of a token's experts are fetched side by side (COMBINE_VEC 4: rows of 16-byte pieces).
template <typename T, int COMBINE_VEC>
__global__ void __launch_bounds__(256) moe_combine_kernel(float* __restrict__ residual, const float* __restrict__ y, const T* __restrict__ h,
                                                          const int* __restrict__ place_of, const float* __restrict__ weights, int top, int W) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const int i = (blockIdx.y * blockDim.x + threadIdx.x) * COMBINE_VEC;
    if (i >= W) return;
    float sum[COMBINE_VEC] = {};
    for (int k = 0; k < top; ++k) {
        const int p = place_of[(size_t)t * top + k];
        const float wk = weights ? weights[(size_t)t * top + k] : 1.f;   // (no weights: they were put on the experts' inputs)
        float v[COMBINE_VEC];
        if (p >= 0) {
            if (COMBINE_VEC == 4) {
                const float4 q = *reinterpret_cast<const float4*>(y + (size_t)p * W + i);
                v[0] = q.x; v[1 % COMBINE_VEC] = q.y; v[2 % COMBINE_VEC] = q.z; v[3 % COMBINE_VEC] = q.w;
            } else {
                v[0] = y[(size_t)p * W + i];
            }
        } else {
#pragma unroll
            for (int j = 0; j < COMBINE_VEC; ++j) v[j] = to_f32(h[(size_t)t * W + i + j]);
        }
#pragma unroll
        for (int j = 0; j < COMBINE_VEC; ++j) sum[j] = fmaf(wk, v[j], sum[j]);
    }
    float* r = residual + (size_t)t * W + i;
    if (COMBINE_VEC == 4) {
        float4 q = *reinterpret_cast<float4*>(r);
        q.x += sum[0]; q.y += sum[1 % COMBINE_VEC]; q.z += sum[2 % COMBINE_VEC]; q.w += sum[3 % COMBINE_VEC];
        *reinterpret_cast<float4*>(r) = q;
    } else {
        r[0] += sum[0];
    }
}

}  // namespace

// logits [N, total + extra]; bias [total] or null; gates [N, extra] (extra 0: none).
LLMIE_API int llmie_moe_route(const float* logits, const float* correction, int* ids, float* weights, int N, int total, int top, int scoring,
                              const float* bias, int extra, float* gates, cudaStream_t s) {
    if (N <= 0) return 0;
    if (total <= 0 || total > 32 * ROUTE_MAX_PER_LANE || top <= 0 || top > total || extra < 0 || (extra && !gates)) return LLMIE_ERR_BAD_ARGUMENT;
    const int per_lane = route_per_lane(total);
    auto kernel = per_lane == 1 ? moe_route_kernel<1> : (per_lane == 4 ? moe_route_kernel<4> : moe_route_kernel<ROUTE_MAX_PER_LANE>);
    return launch_kernel(kernel, dim3((N + 3) / 4), dim3(128), 0, s, logits, correction, ids, weights, N, total, top, scoring, bias, extra,
                         gates);
}

template <typename T, bool EARLY>
static int launch_router_as(const void* h, const void* w, const float* correction, int* ids, float* weights, int N, int K, int total, int top, int scoring,
                            const float* bias, int extra, float* gates, int at_rest, size_t smem, int threads, cudaStream_t s) {
    if (smem > 48 * 1024) {
        static OncePerDevice granted;
        if (const int rc = grant_shared(granted, moe_router_kernel<T, EARLY>, 200 * 1024)) return rc;
    }
    return launch_kernel(moe_router_kernel<T, EARLY>, dim3(N), dim3(threads), smem, s, (const T*)h, (const T*)w, correction, ids, weights, K, total, top, scoring,
                         bias, extra, gates, at_rest);
}

template <typename T>
static int launch_router(const void* h, const void* w, const float* correction, int* ids, float* weights, int N, int K, int total, int top, int scoring,
                         const float* bias, int extra, float* gates, int at_rest, size_t smem, cudaStream_t s) {
    constexpr int VN = Vec16<T>::N, WARPS = ROUTER_THREADS / 32;
    const bool vec = K % VN == 0 && ((uintptr_t)h & 15) == 0 && ((uintptr_t)w & 15) == 0;
    const int pieces = (total + extra + WARPS - 1) / WARPS * ((K + 32 * VN - 1) / (32 * VN));
    const bool few = N <= 148;
#define LLMIE_ROUTER_ARGS(THREADS) h, w, correction, ids, weights, N, K, total, top, scoring, bias, extra, gates, at_rest, smem, THREADS, s
    if (vec && few && pieces <= ROUTER_EARLY) return launch_router_as<T, true>(LLMIE_ROUTER_ARGS(ROUTER_THREADS));
    return launch_router_as<T, false>(LLMIE_ROUTER_ARGS(few ? ROUTER_THREADS : 256));
#undef LLMIE_ROUTER_ARGS
}

// ids, weights [N, top] from the rows h [N, K] and the router's matrix w [total + extra, K] of the same type (float or bfloat16): the product in
// 32-bit and the choice, one launch. at_rest: w may be read before the kernels ahead have finished. The row and the logits must fit the shared memory (K + total floats: up to about 50,000).
LLMIE_API int llmie_moe_router(const void* h, const void* w, const float* correction, int* ids, float* weights, int N, int K, int total, int top,
                               int scoring, const float* bias, int extra, float* gates, int at_rest, int dtype, cudaStream_t s) {
    if (N <= 0) return 0;
    if (K <= 0 || total <= 0 || total > 32 * ROUTE_MAX_PER_LANE || top <= 0 || top > total || extra < 0 || (extra && !gates)) return LLMIE_ERR_BAD_ARGUMENT;
    const size_t smem = ((size_t)((K + 3) & ~3) + total + extra) * sizeof(float);
    if (smem > 200 * 1024) return LLMIE_ERR_BAD_ARGUMENT;
    if (dtype == DT_F32) return launch_router<float>(h, w, correction, ids, weights, N, K, total, top, scoring, bias, extra, gates, at_rest, smem, s);
    return launch_router<bf16>(h, w, correction, ids, weights, N, K, total, top, scoring, bias, extra, gates, at_rest, smem, s);
}

// Rows per tile of the grouped product on the CUDA cores for rows of K numbers: as many as fit the shared memory, at most MOE_TM;
// 0: the rows are too long for it.
LLMIE_API int llmie_moe_tile_rows(int K) {
    if (K <= 0) return 0;
    const long long fit = MOE_ROWS_SMEM / ((long long)K * 4);
    return (int)(fit > MOE_TM ? MOE_TM : fit);
}

// tile_rows: the most places of a tile (what the product that follows wants: llmie_moe_tile_rows(K), or 128 for the tensor cores).
LLMIE_API int llmie_moe_sort(const int* ids, int pairs, int E, int tile_rows, int* offsets, int* perm, int* place_of, int* tiles, int max_tiles,
                             cudaStream_t s) {
    if (pairs <= 0) return 0;
    if (E <= 0 || E > SORT_MAX_EXPERTS || max_tiles <= 0 || tile_rows <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    return launch_kernel(moe_sort_kernel, dim3(1), dim3(pairs <= 512 ? 128 : SORT_THREADS), 0, s, ids, pairs, E, tile_rows, offsets, perm, place_of, tiles, max_tiles);
}

template <typename T, typename TO, bool GATED>
static int launch_moe_rows(const void* x, const int* row_map, int row_div, const void* w, const int* offsets, const int* tiles, int max_tiles, void* out,
                           int F, int K, int tile_rows, const float* row_scale, float limit, float alpha, float shift, cudaStream_t s) {
    const size_t smem = (size_t)tile_rows * K * sizeof(float);
    static size_t allowed = 48 * 1024;
    if (smem > allowed) {
        cudaError_t e = cudaFuncSetAttribute(moe_rows_kernel<T, TO, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOE_ROWS_SMEM);
        if (e != cudaSuccess) return (int)e;
        allowed = MOE_ROWS_SMEM;
    }
    const dim3 grid((F + MOE_COLS - 1) / MOE_COLS, max_tiles);
    return launch_kernel(moe_rows_kernel<T, TO, GATED>, grid, dim3(256), smem, s, (const T*)x, row_map, row_div, (const T*)w, offsets, tiles, (TO*)out, F, K,
                         tile_rows, row_scale, limit, alpha, shift);
}

// gated != 0: w [E][2 F][K], out [places][F] of the storage type; else w [E][F][K], out [places][F] float. tile_rows as given to the sort.
// row_scale [pairs] or null: a weight on every pair's input row (needs row_map); limit > 0: the clamped unit (see the kernel).
LLMIE_API int llmie_moe_gemm(const void* x, const int* row_map, int row_div, const void* w, const int* offsets, const int* tiles, int max_tiles,
                             void* out, int F, int K, int gated, int tile_rows, const float* row_scale, float limit, float alpha, float shift, int dtype,
                             cudaStream_t s) {
    if (max_tiles <= 0) return 0;
    if (F <= 0 || K <= 0 || max_tiles > 65535 || (row_map && row_div <= 0) || tile_rows <= 0 || tile_rows > MOE_TM || tile_rows > llmie_moe_tile_rows(K))
        return LLMIE_ERR_BAD_ARGUMENT;
    if (dtype == DT_F32) {
        if (gated) return launch_moe_rows<float, float, true>(x, row_map, row_div, w, offsets, tiles, max_tiles, out, F, K, tile_rows, row_scale, limit, alpha, shift, s);
        return launch_moe_rows<float, float, false>(x, row_map, row_div, w, offsets, tiles, max_tiles, out, F, K, tile_rows, row_scale, limit, alpha, shift, s);
    }
    if (gated) return launch_moe_rows<bf16, bf16, true>(x, row_map, row_div, w, offsets, tiles, max_tiles, out, F, K, tile_rows, row_scale, limit, alpha, shift, s);
    return launch_moe_rows<bf16, float, false>(x, row_map, row_div, w, offsets, tiles, max_tiles, out, F, K, tile_rows, row_scale, limit, alpha, shift, s);
}

// xs [pairs][K] bfloat16 (K a multiple of 8, 16-byte aligned rows): the tokens' rows in the order of the sort.
LLMIE_API int llmie_moe_gather(const void* x, const int* perm, const int* offsets, int E, int top, void* xs, int pairs, int K, const float* row_scale,
                               cudaStream_t s) {
    if (pairs <= 0) return 0;
    if (K <= 0 || K % 8 || top <= 0 || ((uintptr_t)x & 15) || ((uintptr_t)xs & 15)) return LLMIE_ERR_BAD_ARGUMENT;
    return launch_kernel(moe_gather_kernel, dim3(pairs), dim3(K / 8 < 256 ? (K / 8 < 32 ? 32 : K / 8) : 256), 0, s, (const bf16*)x, perm, offsets, E, top,
                         (bf16*)xs, K, row_scale);
}

LLMIE_API int llmie_moe_combine(float* residual, const float* y, const void* h, const int* place_of, const float* weights, int N, int top, int W,
                                int dtype, cudaStream_t s) {
    if (N <= 0) return 0;
    if (top <= 0 || W <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    const bool vec = W % 4 == 0 && (((uintptr_t)residual | (uintptr_t)y) & 15) == 0;
    const int per = vec ? 4 : 1;
    int threads = 32;
    while (threads < 256 && threads * per < W) threads *= 2;
    const dim3 grid(N, (W + threads * per - 1) / (threads * per));
    if (grid.y > 65535) return LLMIE_ERR_BAD_ARGUMENT;
    if (dtype == DT_F32) {
        if (vec) return launch_kernel(moe_combine_kernel<float, 4>, grid, dim3(threads), 0, s, residual, y, (const float*)h, place_of, weights, top, W);
        return launch_kernel(moe_combine_kernel<float, 1>, grid, dim3(threads), 0, s, residual, y, (const float*)h, place_of, weights, top, W);
    }
    if (vec) return launch_kernel(moe_combine_kernel<bf16, 4>, grid, dim3(threads), 0, s, residual, y, (const bf16*)h, place_of, weights, top, W);
    return launch_kernel(moe_combine_kernel<bf16, 1>, grid, dim3(threads), 0, s, residual, y, (const bf16*)h, place_of, weights, top, W);
}
