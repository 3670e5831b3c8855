// pair32.cuh -- two FP32 lattice nodes in one register pair.
//
// sm_100 executes paired FP32 add / multiply / fused multiply-add
// (__fadd2_rn, __fmul2_rn, __ffma2_rn) at the rate of one scalar instruction,
// so the collision of two nodes written with this type issues about half the
// arithmetic instructions of two scalar collisions.  Every paired operation
// rounds each half as the scalar IEEE operation does; divisions and absolute
// values stay scalar per half.  Used for the FP32-arithmetic kernels (FP32,
// FP16 and BF16 storage).
#pragma once

#include <cuda_runtime.h>

#include "collision_math16.cuh"

namespace vfb
{

struct F2 {
    float2 v;
    F2() = default;
    __host__ __device__ __forceinline__ F2(float s) : v(make_float2(s, s)) {}
    __host__ __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
};

template <>
struct ScalarOf<F2> {
    using type = float;
};

#ifdef __CUDACC__
__device__ __forceinline__ F2 pairOf(float2 x)
{
    F2 r;
    r.v = x;
    return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return pairOf(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return pairOf(__fmul2_rn(a.v, b.v)); }
// negation and subtraction as one paired multiply / multiply-add by -1 (exact)
__device__ __forceinline__ F2 operator-(F2 a) { return pairOf(__fmul2_rn(a.v, make_float2(-1.0f, -1.0f))); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return pairOf(__ffma2_rn(b.v, make_float2(-1.0f, -1.0f), a.v)); }
__device__ __forceinline__ F2 operator/(F2 a, F2 b) { return pairOf(make_float2(a.v.x / b.v.x, a.v.y / b.v.y)); }
__device__ __forceinline__ F2& operator+=(F2& a, F2 b)
{
    a = a + b;
    return a;
}
__device__ __forceinline__ F2& operator-=(F2& a, F2 b)
{
    a = a - b;
    return a;
}
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) { return pairOf(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ F2 fabs(F2 a) { return pairOf(make_float2(fabsf(a.v.x), fabsf(a.v.y))); }

#ifdef __CUDA_ARCH__
template <>
__device__ __forceinline__ F2 limiterReciprocal<F2>(F2 x)
{
    return F2(approximateReciprocal(x.v.x), approximateReciprocal(x.v.y));
}
template <>
__device__ __forceinline__ F2 reciprocal<F2>(F2 x)
{
    const F2 r = limiterReciprocal(x);
    return fma(fma(-x, r, F2(1.0f)), r, r);
}
#endif
#endif

#ifdef __CUDA_ARCH__
template <>
__device__ __forceinline__ F2 termwise::limiterQuotient<F2>(F2 x, F2 y)
{
    return F2(__fdividef(x.v.x, y.v.x), __fdividef(x.v.y, y.v.y));
}
#endif

// K17 rates of a launch duplicated into both halves
inline K17Rates<F2> pairRates(const K17Rates<float>& r)
{
    K17Rates<F2> p;
#define VFB_PAIR(name) p.name = F2(r.name);
    VFB_K17_RATES(VFB_PAIR)
#undef VFB_PAIR
    return p;
}

inline termwise::Rates<F2> pairRates(const termwise::Rates<float>& r)
{
    termwise::Rates<F2> p;
#define VFB_PAIR(name) p.name = F2(r.name);
    VFB_K17_TERM_RATES(VFB_PAIR)
#undef VFB_PAIR
    return p;
}

} // namespace vfb
