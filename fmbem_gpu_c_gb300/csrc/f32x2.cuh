// Packed FP32 arithmetic: two FP32 numbers in a 64-bit register, one instruction for both (the FP32
// pipes' rate, half the issue slots).  Each half rounds as the scalar operation.
#pragma once
#include <cuda_runtime.h>

namespace fmm {

typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_parts(f2 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f2 f2_swap(f2 a)
{
    const float2 v = f2_parts(a);
    return f2_pack(v.y, v.x);
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a - b
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_fma(b, 0xbf800000bf800000ull, a); }

} // namespace fmm
