// out[m, n] (+)= sum_k x[m, k] * w[n, k] for FEW rows m (a decode batch): the weights stream through the
// 5th-generation tensor cores of sm_100a at memory speed.
//
// The product is computed transposed ("swap A/B"): a tile of 128 weight rows is the M side of
// tcgen05.mma (cta_group::1, kind::f16, bfloat16 in, 32-bit accumulate), the TN <= 64 token rows are its
// N side, so no tensor-core work is wasted on padding tokens up to 128. Operands reach shared memory by
// TMA (cp.async.bulk.tensor, 128-byte swizzle, no multicast) through a ring of STAGES buffers guarded by
// mbarriers; the accumulator D[128 x TN] lives in tensor memory and is read back with tcgen05.ld.
//
//   warp 0, one lane   producer: waits for a free stage, arms its barrier with the byte count, issues the
//                      two TMA loads (weight tile 128 x 64, token tile TN x 64; rows or columns outside the
//                      matrices arrive as zeros)
//   warp 1, one lane   issues 4 MMAs (K = 16 each) per stage, commits the stage back to the producer,
//                      and after the last stage commits the accumulator barrier
//   all 4 warps        epilogue: each thread owns one weight row n (TMEM lane) and TN token columns;
//                      it stores, or adds with red.global.add.f32 when the K range is split over blocks
//
// grid = (ceil(N / 128), ceil(M / TN), k_splits). Splitting K gives small matrices enough blocks to pull
// the whole memory system; the partial sums meet in the float32 output by atomic addition, which is
// also how a projection adds itself into the residual stream without a separate kernel. A bias per output is added once, by the
// blocks of the first K range.
//
// Stored results (bfloat16, or float32 that is not added to anything) come from the CLUSTER form: the blocks of a tile's K ranges are a
// thread-block cluster; each puts its sums into its own shared memory, and every block adds up its share of the tile from all of them, first to
// last, with the bias, rounds once and stores. No zeroed output, no second kernel that rounds, and the bits of a row do
// not depend on the order in which blocks finish. A launch of few rows is bound by latency: the library's product of 1 to 16 rows, which
// stood here, cannot start its loads before the kernel ahead has ended nor let the kernel behind fetch its own.
// Measured behind a norm (us, the library's product / this one): 896 x 896 at 1 and 16 rows 6.2 / 4.7 and 5.7 / 5.1, 6,336 x 2,048 9.6 / 8.2 and
// 9.8 / 8.7; 32 outputs of 1,024 in float32, a block alone / eight 8.2 / 4.2. (An activation or a gated unit as its epilogue came out no faster than the
// split-K form with the activation kernel behind it: 4,864 x 896, one row, 7.4 / 6.9.)
//
// Every wait on an mbarrier is bounded: after SPIN_LIMIT polls the block records an error in
// `error_flag`, stops issuing work, lets the copies it started land (again bounded), frees its tensor
// memory and returns. The host reads the flag and raises.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128, BK = 64, STAGES = 4, UMMA_K = 16;

// How a block's sums leave it: added to (or stored in) the float32 output by itself, or through its cluster as float32 or bfloat16.
enum { BY_ITSELF = 0, CLUSTER_F32 = 1, CLUSTER_BF16 = 2 };
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
// 16 bytes of another block's shared memory, at the address that they have in this one's
__device__ __forceinline__ float4 of_block(uint32_t own_address, int rank) {
    float4 v;
    asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %4, %5;\n ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n}\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(own_address), "r"(rank) : "memory");
    return v;
}

template <int TN, bool BIAS, int FORM>
__global__ void __launch_bounds__(128) gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                                                      void* __restrict__ out_base, int ldo, int M, int N, int K, int kb_per_split,
                                                      int accumulate, int* error_flag, const bf16* __restrict__ bias, int at_rest) {
    using Out = typename std::conditional<FORM == CLUSTER_BF16, bf16, float>::type;
    Out* __restrict__ out = static_cast<Out*>(out_base);
    constexpr int W_BYTES = BM * BK * 2, X_BYTES = TN * BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    constexpr int COLS = TN < 32 ? 32 : TN;  // tensor-memory columns: a power of two, at least 32
    extern __shared__ unsigned char raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* accum = empty + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* issued = abort_flag + 1;
    float* sums = reinterpret_cast<float*>(tiles);   // cluster forms: [token][128], over the ring once its MMAs are done
    (void)sums;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * BM, m0 = blockIdx.y * TN;
    const int nkb = (K + BK - 1) / BK;
    const int kb0 = FORM == BY_ITSELF ? blockIdx.z * kb_per_split : nkb * blockIdx.z / gridDim.z;
    const int kb1 = FORM == BY_ITSELF ? min(nkb, kb0 + kb_per_split) : nkb * (blockIdx.z + 1) / gridDim.z;
    const int iters = kb1 - kb0;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        mbar_init(accum, 1);
        *abort_flag = 0;
        *issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();  // lane 0 comes back from the initialisation above: the allocation is a warp-wide instruction
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "n"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    pdl_trigger();
    if (warp == 0 && lane == 0) {
        if constexpr (FORM != BY_ITSELF) pdl_wait_unless(at_rest);
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&tmap_w) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&tmap_x) : "memory");
        // The weights do not depend on the kernel before this one: the first stages' weight tiles are on their way
        // before the wait; the token tiles, which that kernel wrote, follow after it.
        const auto load_w = [&](unsigned char* to, int it, uint64_t* bar) {
            tma_load_2d(to, &tmap_w, (kb0 + it) * BK, n0, bar);
        };
        const int early = min(iters, STAGES);
        constexpr uint32_t tx = STAGE_BYTES;
        for (int it = 0; it < early; ++it) {
            mbar_expect_tx(full + it, tx);
            load_w(tiles + it * STAGE_BYTES, it, full + it);
            *issued = it + 1;
        }
        pdl_wait();
        for (int it = 0; it < early; ++it) tma_load_2d(tiles + it * STAGE_BYTES + W_BYTES, &tmap_x, (kb0 + it) * BK, m0, full + it);
        for (int it = early; it < iters; ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(empty + s, ((it / STAGES) & 1) ^ 1, abort_flag, error_flag, 1)) break;
            unsigned char* st = tiles + s * STAGE_BYTES;
            mbar_expect_tx(full + s, tx);
            load_w(st, it, full + s);
            tma_load_2d(st + W_BYTES, &tmap_x, (kb0 + it) * BK, m0, full + s);
            *issued = it + 1;
        }
    } else if (warp == 1 && lane == 0) {
        // instruction descriptor: D float32, A and B bfloat16, both K-major, N = TN, M = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        bool ok = true;
        for (int it = 0; it < iters && ok; ++it) {
            const int s = it % STAGES;
            ok = mbar_wait(full + s, (it / STAGES) & 1, abort_flag, error_flag, 2);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t a_addr = smem_u32(tiles + s * STAGE_BYTES);
            const uint64_t a_desc = umma_desc(a_addr), b_desc = umma_desc(a_addr + W_BYTES);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
                umma_bf16(tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, (it > 0 || k > 0) ? 1u : 0u);  // +32 bytes per K step
            umma_commit(empty + s);
        }
        if (ok) umma_commit(accum);
    }
    __syncwarp();
    pdl_wait();  // every thread: the epilogue writes where the kernel before may still read or write
    const bool done = __all_sync(0xffffffffu, mbar_wait(accum, 0, abort_flag, error_flag, 3));  // uniform per warp: tcgen05.ld is warp-wide
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if constexpr (FORM != BY_ITSELF) {
        const int rows = min(TN, M - m0), S = gridDim.z, rank = blockIdx.z;
        if (done) {   // (this block's MMAs are over: its ring is free)
#pragma unroll
            for (int c = 0; c < TN; c += 16) {
                if (c >= rows) break;
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c + j < rows) sums[(c + j) * BM + tid] = __uint_as_float(v[j]);
            }
        }
        cluster_arrive();   // (a block that gave up takes part all the same: the results are not valid then, and the host is told)
        cluster_wait();
        // four neighbouring outputs of a row to a thread, the tile's pieces dealt out over the blocks in runs
        const int pieces = rows * (BM / 4), share = (pieces + S - 1) / S, end = min(pieces, (rank + 1) * share);
        const uint32_t base = smem_u32(sums);
        for (int e = rank * share + tid; e < end; e += 128) {
            const int m = e / (BM / 4), o = e % (BM / 4) * 4, n = n0 + o;
            if (n >= N) continue;
            float4 part[8];
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (b < S) part[b] = of_block(base + e * 16, b);
            float t[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
            for (int b = 1; b < 8; ++b)
                if (b < S) { t[0] += part[b].x; t[1] += part[b].y; t[2] += part[b].z; t[3] += part[b].w; }
            const size_t at = (size_t)(m0 + m) * ldo + n;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (BIAS) t[j] += n + j < N ? to_f32(bias[n + j]) : 0.f;
            }
            if ((ldo & 3) == 0 && n + 4 <= N) {
                store4(out + at, t);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N) out[at + j] = from_f32<Out>(t[j]);
            }
        }
        cluster_arrive();   // nobody's shared memory goes away while it is read
        cluster_wait();
    } else if (done) {
        const int n = n0 + warp * 32 + lane;
        const int rows = min(TN, M - m0);
        float add = 0.f;
        if constexpr (BIAS) add = (n < N && blockIdx.z == 0) ? to_f32(bias[n]) : 0.f;
#pragma unroll
        for (int c = 0; c < TN; c += 16) {
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (n < N) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int m = c + j;
                    if (m < rows) {
                        float* dst = out + (size_t)(m0 + m) * ldo + n;
                        if (accumulate) atomicAdd(dst, BIAS ? __uint_as_float(v[j]) + add : __uint_as_float(v[j]));
                        else *dst = BIAS ? __uint_as_float(v[j]) + add : __uint_as_float(v[j]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (!done && tid == 0) {
        // gave up somewhere: let the copies that were started land before the block's shared memory goes away
        const int n_issued = *issued;
        for (int it = max(0, n_issued - STAGES); it < n_issued; ++it) {
            for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
                if (mbar_try_wait(full + it % STAGES, (it / STAGES) & 1)) break;
                __nanosleep(40);
            }
        }
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(COLS) : "memory");
}

// ------------------------------------------------------------------------------------------------ host side
struct Call {
    void* out;
    int ldo, M, N, K, k_splits, accumulate;
    int* error_flag;
    const bf16* bias;
    int at_rest;
};

template <int TN, bool BIAS, int FORM>
int launch_as(const CUtensorMap& mw, const CUtensorMap& mx, const Call& c, cudaStream_t s) {
    constexpr size_t smem = (size_t)STAGES * (BM * BK * 2 + TN * BK * 2) + 1024 + 256;
    static OncePerDevice granted;
    const int rc = grant_shared(granted, gemm_tc_kernel<TN, BIAS, FORM>, (int)smem);
    if (rc) return rc;
    const int nkb = (c.K + BK - 1) / BK;
    const int per = (nkb + c.k_splits - 1) / c.k_splits;
    const int splits = FORM == BY_ITSELF ? (nkb + per - 1) / per : c.k_splits;  // no empty split; a cluster is whole: the host asks for no more blocks than K has pieces
    const dim3 grid((c.N + BM - 1) / BM, (c.M + TN - 1) / TN, splits);
    if constexpr (FORM == BY_ITSELF)
        return launch_kernel(gemm_tc_kernel<TN, BIAS, FORM>, grid, dim3(128), smem, s, mw, mx, c.out, c.ldo, c.M, c.N, c.K, per, c.accumulate,
                             c.error_flag, c.bias, 1);
    else
        return launch_cluster(gemm_tc_kernel<TN, BIAS, FORM>, grid, dim3(128), dim3(1, 1, splits), smem, s, mw, mx, c.out, c.ldo, c.M, c.N, c.K, per,
                              c.accumulate, c.error_flag, c.bias, c.at_rest);
}

template <int TN, int FORM>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Call& c, cudaStream_t s) {
    return c.bias ? launch_as<TN, true, FORM>(mw, mx, c, s) : launch_as<TN, false, FORM>(mw, mx, c, s);
}

template <int FORM>
int run(const bf16* x, int ldx, const bf16* w, const Call& c, cudaStream_t s) {
    if (c.M <= 0 || c.N <= 0) return 0;
    if (c.K <= 0 || c.K % 8 || ((uintptr_t)w & 15) || ((uintptr_t)x & 15) || ldx < c.K || ldx % 8 || !c.error_flag || c.ldo < c.N)
        return LLMIE_ERR_BAD_ARGUMENT;
    const int TN = c.M <= 16 ? 16 : (c.M <= 32 ? 32 : 64);
    CUtensorMap mw, mx;
    int rc = tensor_map(w, c.N, c.K, BM, &mw);
    if (rc) return rc;
    rc = tensor_map(x, c.M, c.K, TN, &mx, ldx);
    if (rc) return rc;
    if (TN == 16) return launch<16, FORM>(mw, mx, c, s);
    if (TN == 32) return launch<32, FORM>(mw, mx, c, s);
    return launch<64, FORM>(mw, mx, c, s);
}

}  // namespace

// x [M, K] and w [N, K] bfloat16 row-major (K a multiple of 8, bases 16-byte aligned), out float32 with row stride ldo.
// accumulate = 0 needs k_splits = 1 and stores; accumulate = 1 adds atomically into what `out` holds. bias: [N] bfloat16 or null.
LLMIE_API int llmie_gemm_tc(const bf16* x, const bf16* w, float* out, int ldo, int M, int N, int K, int k_splits, int accumulate,
                            int* error_flag, const bf16* bias, cudaStream_t s) {
    if (k_splits < 1 || (!accumulate && k_splits != 1)) return LLMIE_ERR_BAD_ARGUMENT;
    return run<BY_ITSELF>(x, K, w, Call{out, ldo, M, N, K, k_splits, accumulate, error_flag, bias, 1}, s);
}

// The same, stored: out [M, N] float32 or bfloat16 (contiguous), x with rows ldx elements apart (a multiple of 8), the K range over a
// cluster of `blocks` (1, 2, 4 or 8, no more than K has pieces of 64). at_rest: w lies at rest and
// may be fetched ahead of the kernel before.
LLMIE_API int llmie_gemm_tc_store(const bf16* x, int ldx, const bf16* w, void* out, int out_dt, int M, int N, int K, int blocks, int* error_flag,
                                  const bf16* bias, int at_rest, cudaStream_t s) {
    const int pieces = (K + BK - 1) / BK;
    if (blocks < 1 || blocks > 8 || (blocks & (blocks - 1)) || blocks > pieces || ((uintptr_t)out & 15))
        return LLMIE_ERR_BAD_ARGUMENT;
    const Call c{out, N, M, N, K, blocks, 0, error_flag, bias, at_rest};
    return out_dt == DT_BF16 ? run<CLUSTER_BF16>(x, ldx, w, c, s) : run<CLUSTER_F32>(x, ldx, w, c, s);
}
