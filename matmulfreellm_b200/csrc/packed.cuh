// Rows of 16-bit activations held as packed pairs: widening, rounding, exact sums of squares, codes.
#pragma once
#include "common.cuh"

namespace {

// asynchronous 16-byte copy global -> shared memory (no register staging) and its group bookkeeping
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <typename T> __device__ __forceinline__ float2 widen(uint32_t u) {
    if constexpr (cuda::std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&u));
    else return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
template <typename T> __device__ __forceinline__ uint32_t narrow(float2 v) {
    if constexpr (cuda::std::is_same<T, __half>::value) {
        const __half2 h = __floats2half2_rn(v.x, v.y);
        return *reinterpret_cast<const uint32_t*>(&h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
}
// s0 / s1 += squares of a packed pair (bf16: the fp64 operands are assembled from the bits, as sumsq_rounded does)
template <typename T> __device__ __forceinline__ void sumsq_pair(uint32_t u, double& s0, double& s1) {
    if constexpr (cuda::std::is_same<T, __half>::value) {
        const float2 f = widen<T>(u);
        s0 = fma((double)f.x, (double)f.x, s0);
        s1 = fma((double)f.y, (double)f.y, s1);
    } else {
        const double d0 = __hiloint2double((int)(((u & 0x7fffu) << 13) + 0x38000000u), 0);
        const double d1 = __hiloint2double((int)(((u >> 3) & 0x0fffe000u) + 0x38000000u), 0);
        s0 = fma(d0, d0, s0);
        s1 = fma(d1, d1, s1);
    }
}
__device__ __forceinline__ float2 mul2(float2 a, float b) { return __fmul2_rn(a, make_float2(b, b)); }
__device__ __forceinline__ void lds8(const float* p, float2 (&w)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    w[0] = make_float2(a.x, a.y); w[1] = make_float2(a.z, a.w);
    w[2] = make_float2(b.x, b.y); w[3] = make_float2(b.z, b.w);
}
// int8 codes of four values (already normalised and weighted) with scale s, as one word.  |y * s| <= 127 (1 + 2^-23): no clamp;
// adding 1.5 * 2^23 leaves the code, rounded to nearest even, in the low byte.  Scalar on purpose: a packed multiply feeding a
// packed add can be merged into one rounding.
__device__ __forceinline__ uint32_t codes4(float2 y0, float2 y1, float s) {
    const int a = __float_as_int(__fadd_rn(__fmul_rn(y0.x, s), 12582912.0f)), b = __float_as_int(__fadd_rn(__fmul_rn(y0.y, s), 12582912.0f));
    const int c = __float_as_int(__fadd_rn(__fmul_rn(y1.x, s), 12582912.0f)), d = __float_as_int(__fadd_rn(__fmul_rn(y1.y, s), 12582912.0f));
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

}  // namespace
