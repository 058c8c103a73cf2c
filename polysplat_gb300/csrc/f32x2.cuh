// Pairs of floats in one 64-bit register and the paired FP32 instructions of
// sm_100 and later.  Each half rounds like the scalar instruction, so a pair
// gives the bits of two scalar operations for one issue slot.
#pragma once

#include <stdint.h>

namespace gsr {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pair(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void split(f32x2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ float lo_of(f32x2 v)
{
    float lo, hi;
    split(v, lo, hi);
    return lo;
}
__device__ __forceinline__ float hi_of(f32x2 v)
{
    float lo, hi;
    split(v, lo, hi);
    return hi;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// ex2.approx of both halves
__device__ __forceinline__ f32x2 ex2_2(f32x2 v)
{
    float a, b;
    split(v, a, b);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(a));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(b));
    return pair(a, b);
}
__device__ __forceinline__ float rcp_approx_ftz(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// max that keeps a NaN, as a chain of comparisons does
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

}  // namespace gsr
