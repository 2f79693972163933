// What the recurrences' kernels share: multiply-adds on pairs of floats, and sums over the PARTS lanes that share a column of a state.
#pragma once

#include <cuda_runtime.h>

// two 32-bit multiply-adds (multiplications) in one instruction
__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
          "l"(reinterpret_cast<const unsigned long long&>(c)));
    return reinterpret_cast<float2&>(d);
}
__device__ __forceinline__ float2 mul2(const float2& a, const float2& b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
    return reinterpret_cast<float2&>(d);
}

// the sum of v over the group's lanes, in every lane
template <int PARTS> __device__ __forceinline__ float parts_sum(float v) {
#pragma unroll
    for (int o = PARTS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// v[i] is this lane's share of sum i, i < PARTS; lane `part` of the group of PARTS lanes ends with the whole of sum `part`.
// Halves change hands, so PARTS - 1 shuffles serve PARTS sums; each sum is added up in the order of parts_sum.
template <int PARTS>
__device__ __forceinline__ float parts_scatter(float* v, int part) {
#pragma unroll
    for (int o = PARTS / 2; o > 0; o >>= 1) {
        const bool up = part & o;
#pragma unroll
        for (int t = 0; t < o; ++t) {
            const float give = up ? v[t] : v[t + o], keep = up ? v[t + o] : v[t];
            v[t] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}
