// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) on the CUDA cores, 32-bit multiply-add, one fixed order over K.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no reduced-precision mode),
// and it also takes bfloat16 inputs (32-bit accumulate) for shapes the tensor-core kernels refuse.
//
// The order: K is cut into 1, 2, 4 or 8 slices of equal length (a multiple of 32, chosen by K alone). Within a slice the even and the odd
// k are two chains of fused multiply-adds; a slice is even + odd, and the slices are added first to last. Every kernel below keeps
// it, so a token's result does not depend on M, on where its row lies in the batch or on which kernel ran. Two chains because sm_100
// has a packed multiply-add on two floats (fma.rn.f32x2) whose operands, k and k + 1 of a row, lie side by side in memory; slices
// because a decoded token's product would otherwise be one long chain on a few blocks. Both shorten the chains of roundings.
//
//   small_kernel    M <= 16: weights stream at memory speed. A block owns 32 outputs (one per lane) of ONE slice and fetches its
//                   32 rows of it with asynchronous 16-byte copies, up to SMALL_STAGES chunks of 128 k in flight, the first ones
//                   before the kernel ahead has finished (weights at rest); a warp takes up to 4 token rows. The slices of an output are a cluster.
//   tile_kernel     more rows: bound by the multiply-adds. 64 x 64 or 64 x 128 outputs of one slice per block, 8 x 4 or 8 x 8 per
//                   thread, both operands row-major in shared memory (rows 36 floats apart: eight lanes' 16-byte reads fall into
//                   eight different bank groups), so nothing is transposed; the slices of a tile are a cluster, which adds
//                   its partial tiles through distributed shared memory.
//   gemm_simt_kernel  anything else (bfloat16, rows or bases that are not 16-byte aligned).
//
// Measured against gemm_simt_kernel for every shape (rows x outputs x inner, microseconds): 302 x 9728 x 896 198 -> 139 (38 TFLOP/s),
// 302 x 896 x 4864 369 -> 88, 302 x 896 x 896 57 -> 23, 3 x 9728 x 896 91 -> 13, 3 x 896 x 4864 409 -> 12, 3 x 151936 x 896 516 -> 195;
// relative error 5.4e-7 -> 2.0e-7 at an inner size of 896, 1.2e-6 -> 3.2e-7 at 4864.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

struct Slices { int count, length; };
__host__ __device__ inline Slices slices_of(int K) {
    const int n = K <= 256 ? 1 : (K <= 512 ? 2 : (K <= 1024 ? 4 : 8));
    return {n, ((K + n - 1) / n + 31) / 32 * 32};
}

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 16 x 16 threads, 4 x 4 outputs each

template <typename T>
__device__ __forceinline__ void load4(const T* __restrict__ base, int row, int rows, int k, int K, bool vec, float* out) {
    out[0] = out[1] = out[2] = out[3] = 0.f;
    if (row >= rows) return;
    const T* p = base + (size_t)row * K + k;
    if (vec && k + 3 < K) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
        } else {
            const uint2 v = *reinterpret_cast<const uint2*>(p);
            out[0] = __uint_as_float(v.x << 16); out[1] = __uint_as_float(v.x & 0xffff0000u);
            out[2] = __uint_as_float(v.y << 16); out[3] = __uint_as_float(v.y & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (k + i < K) out[i] = to_f32(p[i]);
    }
}

template <typename TI, typename TO>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const TI* __restrict__ A, const TI* __restrict__ W, TO* __restrict__ C,
                                                       int M, int N, int K, int vec, int accumulate, const TI* __restrict__ bias) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lrow = tid >> 2, lk = (tid & 3) * 4;  // each thread stages 4 consecutive k of one row of each tile
    const int slice = slices_of(K).length;
    float total[TM][TN], acc[2][TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[1][i][j] = total[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        float a[4], w[4];
        load4<TI>(A, m0 + lrow, M, k0 + lk, K, vec, a);
        load4<TI>(W, n0 + lrow, N, k0 + lk, K, vec, w);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            As[lk + i][lrow] = a[i];
            Ws[lk + i][lrow] = w[i];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float av[TM], wv[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) wv[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[kk & 1][i][j] = fmaf(av[i], wv[j], acc[kk & 1][i][j]);
        }
        if ((k0 + BK) % slice == 0 || k0 + BK >= K) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float s = acc[0][i][j] + acc[1][i][j];
                    total[i][j] = k0 < slice ? s : total[i][j] + s;
                    acc[0][i][j] = acc[1][i][j] = 0.f;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) {
                TO* dst = C + (size_t)m * N + n;  // with `accumulate` the product is added to what C holds (its only writer is this thread)
                const float v = bias ? total[i][j] + to_f32(bias[n]) : total[i][j];
                *dst = from_f32<TO>(accumulate ? to_f32(*dst) + v : v);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ aligned 32-bit rows
__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {  // zeros where `there` is false (nothing is read)
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// c.x += a.x * b.x, c.y += a.y * b.y
__device__ __forceinline__ void fma2(float2& c, const float2& a, const float2& b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(reinterpret_cast<unsigned long long&>(c))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

struct F32Args {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, accumulate;
    int at_rest;   // W was written before the kernels that may still be running: see pdl_wait_unless
};

__device__ __forceinline__ void put(const F32Args& p, int m, int n, float v) {
    float* dst = p.C + (size_t)m * p.N + n;
    if (p.bias) v += p.bias[n];
    *dst = p.accumulate ? *dst + v : v;
}

constexpr int CHUNK = 128, CHUNK_PITCH = CHUNK + 4, SMALL_STAGES = 5, SMALL_ROWS = 16;

// block (0 .. ceil(M / R) - 1) warps; grid (ceil(N / 32), slices), the slices of 32 outputs one cluster
template <int R>
__global__ void __launch_bounds__(128) small_kernel(F32Args p, int stages) {
    extern __shared__ float4 small_shared[];
    float* ring = reinterpret_cast<float*>(small_shared);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int rows = warps * R, stage_floats = (32 + rows) * CHUNK_PITCH;
    const Slices sl = slices_of(p.K);
    const int n0 = blockIdx.x * 32, slice = blockIdx.y;
    const int k0 = slice * sl.length, k1 = min(p.K, k0 + sl.length);
    const int chunks = (k1 - k0 + CHUNK - 1) / CHUNK;

    auto fetch_weights = [&](int c) {
        float* to = ring + (c % stages) * stage_floats;
        const int k = k0 + c * CHUNK + lane * 4;
        for (int r = warp; r < 32; r += warps)
            copy16(to + r * CHUNK_PITCH + lane * 4, p.W + (size_t)min(n0 + r, p.N - 1) * p.K + min(k, p.K - 4), k < k1 && n0 + r < p.N);
    };
    auto fetch_tokens = [&](int c) {
        float* to = ring + (c % stages) * stage_floats + 32 * CHUNK_PITCH;
        const int k = k0 + c * CHUNK + lane * 4;
        for (int r = warp; r < rows; r += warps)
            copy16(to + r * CHUNK_PITCH + lane * 4, p.A + (size_t)min(r, p.M - 1) * p.K + min(k, p.K - 4), k < k1 && r < p.M);
    };
    pdl_trigger();
    const int early = min(stages, chunks);
    pdl_wait_unless(p.at_rest);
    for (int c = 0; c < early; ++c) fetch_weights(c);   // weights at rest are fetched while the kernel ahead still runs
    pdl_wait();
    for (int c = 0; c < early; ++c) fetch_tokens(c);
    copies_commit();
    float2 acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = make_float2(0.f, 0.f);
    for (int c = 0; c < chunks; ++c) {
        if (c == 0 || c >= early) copies_wait<0>();
        if (c == 0 || c >= early) __syncthreads();
        const float* w = ring + (c % stages) * stage_floats + lane * CHUNK_PITCH;
        const float* x = ring + (c % stages) * stage_floats + (32 + warp * R) * CHUNK_PITCH;
        const int len = min(CHUNK, k1 - k0 - c * CHUNK);
#pragma unroll 8
        for (int k = 0; k < len; k += 4) {
            const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float4 xv = *reinterpret_cast<const float4*>(x + i * CHUNK_PITCH + k);
                fma2(acc[i], make_float2(xv.x, xv.y), make_float2(wv.x, wv.y));
                fma2(acc[i], make_float2(xv.z, xv.w), make_float2(wv.z, wv.w));
            }
        }
        if (c + stages < chunks) {
            __syncthreads();
            fetch_weights(c + stages);
            fetch_tokens(c + stages);
            copies_commit();
        }
    }
    if (sl.count == 1) {
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (warp * R + i < p.M && n0 + lane < p.N) put(p, warp * R + i, n0 + lane, acc[i].x + acc[i].y);
        return;
    }
    __shared__ float part[SMALL_ROWS][32];
#pragma unroll
    for (int i = 0; i < R; ++i) part[warp * R + i][lane] = acc[i].x + acc[i].y;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int m = slice + sl.count * warp; m < p.M; m += sl.count * warps) {   // a row's sum by one warp of one block of the cluster
        float v[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < sl.count) v[s] = *cluster.map_shared_rank(&part[m][lane], s);
        float t = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < sl.count) t += v[s];
        if (n0 + lane < p.N) put(p, m, n0 + lane, t);
    }
    cluster.sync();   // a block's partial sums are read until here
}

constexpr int TILE_M = 64, TILE_K = 32, TILE_PITCH = TILE_K + 4, TILE_STAGES = 3;

// 128 threads: 8 (rows) x 16 (columns); a thread owns rows ty + 8 i and columns tx + 16 j. grid (ceil(N / (16 COLS)), ceil(M / 64), slices)
template <int COLS>
__global__ void __launch_bounds__(128) tile_kernel(F32Args p) {
    constexpr int TILE_N = 16 * COLS, STAGE = (TILE_M + TILE_N) * TILE_PITCH, OUT_PITCH = TILE_N + 4;
    static_assert(TILE_M * OUT_PITCH <= TILE_STAGES * STAGE, "the partial tile takes the ring's place");
    extern __shared__ float4 tile_shared[];
    float* ring = reinterpret_cast<float*>(tile_shared);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const Slices sl = slices_of(p.K);
    const int n0 = blockIdx.x * TILE_N, m0 = blockIdx.y * TILE_M, slice = blockIdx.z;
    const int k0 = slice * sl.length, k1 = min(p.K, k0 + sl.length);
    const int steps = (k1 - k0 + TILE_K - 1) / TILE_K;
    const int frow = tid >> 3, fk = (tid & 7) * 4;   // eight threads fetch a row's 32 k, 16 rows at a time

    auto fetch = [&](int t, bool weights, bool tokens) {
        float* to = ring + (t % TILE_STAGES) * STAGE + frow * TILE_PITCH + fk;
        const int k = k0 + t * TILE_K + fk;
        const bool in = k < k1;
        const int kk = min(k, p.K - 4);
        if (tokens) {
#pragma unroll
            for (int r = 0; r < TILE_M; r += 16)
                copy16(to + r * TILE_PITCH, p.A + (size_t)min(m0 + frow + r, p.M - 1) * p.K + kk, in && m0 + frow + r < p.M);
        }
        if (weights) {
#pragma unroll
            for (int r = 0; r < TILE_N; r += 16)
                copy16(to + (TILE_M + r) * TILE_PITCH, p.W + (size_t)min(n0 + frow + r, p.N - 1) * p.K + kk, in && n0 + frow + r < p.N);
        }
    };
    float2 acc[8][COLS];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[i][j] = make_float2(0.f, 0.f);
    pdl_trigger();
    pdl_wait_unless(p.at_rest);
    for (int t = 0; t < TILE_STAGES - 1; ++t)
        if (t < steps) fetch(t, true, false);
    pdl_wait();
    for (int t = 0; t < TILE_STAGES - 1; ++t) {
        if (t < steps) fetch(t, false, true);
        copies_commit();
    }
    for (int t = 0; t < steps; ++t) {
        copies_wait<TILE_STAGES - 2>();
        __syncthreads();   // stage t has arrived for everyone, and everyone is done with stage t - 1
        if (t + TILE_STAGES - 1 < steps) fetch(t + TILE_STAGES - 1, true, true);
        copies_commit();
        const float* a = ring + (t % TILE_STAGES) * STAGE + ty * TILE_PITCH;
        const float* w = ring + (t % TILE_STAGES) * STAGE + (TILE_M + tx) * TILE_PITCH;
#pragma unroll
        for (int k = 0; k < TILE_K; k += 4) {
            float4 av[8], wv[COLS];
#pragma unroll
            for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * 8 * TILE_PITCH + k);
#pragma unroll
            for (int j = 0; j < COLS; ++j) wv[j] = *reinterpret_cast<const float4*>(w + j * 16 * TILE_PITCH + k);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < COLS; ++j) fma2(acc[i][j], make_float2(av[i].x, av[i].y), make_float2(wv[j].x, wv[j].y));
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < COLS; ++j) fma2(acc[i][j], make_float2(av[i].z, av[i].w), make_float2(wv[j].z, wv[j].w));
        }
    }
    if (sl.count == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int m = m0 + ty + 8 * i, n = n0 + tx + 16 * j;
                if (m < p.M && n < p.N) put(p, m, n, acc[i][j].x + acc[i][j].y);
            }
        return;
    }
    __syncthreads();   // the ring becomes the block's partial tile (every copy into it has landed: the last ones were waited for above)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < COLS; ++j) ring[(ty + 8 * i) * OUT_PITCH + tx + 16 * j] = acc[i][j].x + acc[i][j].y;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int rows = TILE_M / sl.count;   // each block of the cluster adds up its share of the tile's rows
    for (int e = tid; e < rows * (TILE_N / 4); e += 128) {
        const int r = slice * rows + e / (TILE_N / 4), c = e % (TILE_N / 4) * 4;
        if (m0 + r >= p.M) break;
        float4 v[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < sl.count) v[s] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(ring + r * OUT_PITCH + c, s));
        float4 t = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < sl.count) { t.x += v[s].x; t.y += v[s].y; t.z += v[s].z; t.w += v[s].w; }
        const float out[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + c + j < p.N) put(p, m0 + r, n0 + c + j, out[j]);
    }
    cluster.sync();
}

template <typename Kernel>
int launch_sliced(Kernel kernel, dim3 grid, dim3 block, dim3 cluster, size_t smem, cudaStream_t s, const F32Args& p, int stages) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster.x;
    attr[0].val.clusterDim.y = cluster.y;
    attr[0].val.clusterDim.z = cluster.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = llmie_pdl_flag ? 2 : 1;
    if constexpr (std::is_same_v<Kernel, void (*)(F32Args)>) return (int)cudaLaunchKernelEx(&cfg, kernel, p);
    else return (int)cudaLaunchKernelEx(&cfg, kernel, p, stages);
}

template <int R>
int run_small(const F32Args& p, cudaStream_t s) {
    const Slices sl = slices_of(p.K);
    const int warps = (p.M + R - 1) / R, stages = min(SMALL_STAGES, (sl.length + CHUNK - 1) / CHUNK);
    constexpr int most = SMALL_STAGES * (32 + SMALL_ROWS) * CHUNK_PITCH * 4;
    static OncePerDevice granted;
    if (const int rc = grant_shared(granted, small_kernel<R>, most)) return rc;
    return launch_sliced(small_kernel<R>, dim3((p.N + 31) / 32, sl.count), dim3(32 * warps), dim3(1, sl.count, 1),
                         (size_t)stages * (32 + warps * R) * CHUNK_PITCH * 4, s, p, stages);
}

template <int COLS>
int run_tiles(const F32Args& p, cudaStream_t s) {
    constexpr int smem = TILE_STAGES * (TILE_M + 16 * COLS) * TILE_PITCH * 4;
    static OncePerDevice granted;
    if (const int rc = grant_shared(granted, tile_kernel<COLS>, smem)) return rc;
    const Slices sl = slices_of(p.K);
    return launch_sliced(tile_kernel<COLS>, dim3((p.N + 16 * COLS - 1) / (16 * COLS), (p.M + TILE_M - 1) / TILE_M, sl.count), dim3(128),
                         dim3(1, 1, sl.count), smem, s, p, 0);
}

int run_f32(const F32Args& p, cudaStream_t s) {
    // 16 rows: 30 us here, 17 rows: 39 us on tiles (9,728 outputs, inner size 896)
    if (p.M <= SMALL_ROWS) {
        if (p.M == 1) return run_small<1>(p, s);
        if (p.M == 2) return run_small<2>(p, s);
        if (p.M == 3) return run_small<3>(p, s);
        return run_small<4>(p, s);
    }
    // tiles of 128 outputs read 2 floats of shared memory per 8 multiply-adds, tiles of 64 read 3: the wide ones where they give two blocks
    // to every multiprocessor
    const long long wide = (long long)((p.N + 127) / 128) * ((p.M + TILE_M - 1) / TILE_M) * slices_of(p.K).count;
    return wide >= 2 * 148 ? run_tiles<8>(p, s) : run_tiles<4>(p, s);
}

}  // namespace

// in_dtype / out_dtype: 0 float32, 1 bfloat16; bias (or null) in in_dtype; at_rest: W may be read before the kernels ahead have finished. Beyond K the tiles are padded with zeros, which add nothing.
LLMIE_API int llmie_gemm_simt(const void* A, const void* W, void* C, int M, int N, int K, int in_dtype, int out_dtype,
                              int accumulate, const void* bias, int at_rest, cudaStream_t s) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return LLMIE_ERR_BAD_ARGUMENT;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    const int vec = (K % 4 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
    if (in_dtype == DT_F32 && out_dtype == DT_F32) {
        if (vec && (M + TILE_M - 1) / TILE_M <= 65535)
            return run_f32({(const float*)A, (const float*)W, (const float*)bias, (float*)C, M, N, K, accumulate, at_rest}, s);
        gemm_simt_kernel<float, float><<<grid, 256, 0, s>>>((const float*)A, (const float*)W, (float*)C, M, N, K, vec, accumulate, (const float*)bias);
    } else if (in_dtype == DT_BF16 && out_dtype == DT_F32)
        gemm_simt_kernel<bf16, float><<<grid, 256, 0, s>>>((const bf16*)A, (const bf16*)W, (float*)C, M, N, K, vec, accumulate, (const bf16*)bias);
    else if (in_dtype == DT_BF16 && out_dtype == DT_BF16)
        gemm_simt_kernel<bf16, bf16><<<grid, 256, 0, s>>>((const bf16*)A, (const bf16*)W, (bf16*)C, M, N, K, vec, accumulate, (const bf16*)bias);
    else
        return LLMIE_ERR_BAD_ARGUMENT;
    return launch_status();
}
