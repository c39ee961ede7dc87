// Packed FP32x2 arithmetic for sm_100a: two independent nodes' values in one 64-bit register pair,
// every add, multiply and fused multiply-add issued as one instruction for both (sm_100's f32x2
// operations, each lane rounded as the scalar operation).
// The K17 collision is generic over its arithmetic type, so instantiated with f2 it collides two
// nodes per thread at half the instruction count of the arithmetic, each node with the bits of the
// scalar form.
#pragma once

#include <cuda_runtime.h>

#include "k17.cuh"

namespace vfb {

struct f2 {
    float2 v;
    f2() = default;
    __host__ __device__ __forceinline__ f2(float a) : v{ a, a } {}
    __host__ __device__ __forceinline__ f2(float a, float b) : v{ a, b } {}
};

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
#else
__host__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__host__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
#endif
__host__ __device__ __forceinline__ f2 wrap(float2 v) { f2 r; r.v = v; return r; }
__host__ __device__ __forceinline__ f2 operator+(f2 a, f2 b) { return wrap(add2(a.v, b.v)); }
// a - b = b * (-1) + a: the product is exact, so one rounding as in the scalar subtraction
__host__ __device__ __forceinline__ f2 operator-(f2 a, f2 b) { return wrap(fma2(b.v, make_float2(-1.0f, -1.0f), a.v)); }
__host__ __device__ __forceinline__ f2 operator*(f2 a, f2 b) { return wrap(mul2(a.v, b.v)); }
__host__ __device__ __forceinline__ f2 operator-(f2 a) { return f2(-a.v.x, -a.v.y); }
__host__ __device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) { return wrap(fma2(a.v, b.v, c.v)); }

__host__ __device__ __forceinline__ f2 rho_rcp(f2 x) { return f2(k17detail::rho_rcp(x.v.x), k17detail::rho_rcp(x.v.y)); }
__host__ __device__ __forceinline__ void limiter_inverses(const f2 (&m)[7], const float (&q)[7], f2 (&iv)[7])
{
#pragma unroll
    for (int i = 0; i < 7; ++i)
        iv[i] = f2(k17detail::fast_rcp(rn_add(fabsf(m[i].v.x), q[i])), k17detail::fast_rcp(rn_add(fabsf(m[i].v.y), q[i])));
}

} // namespace vfb
