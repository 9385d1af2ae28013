// Float-float arithmetic for the FP64-quality translations on the FP32 pipes (GB300's FP64
// rate is a 64th of its FP32 rate).  A value is the unevaluated sum hi + lo of two FP32 numbers
// with |lo| <= ulp(hi) / 2: about 48 significant bits, with FP32's exponent range.
//
// The operations are built from the classical error-free transformations: Knuth's TwoSum
// (s + e = a + b exactly) and Dekker's FastTwoSum (the same for |a| >= |b|), combined as the
// double-word addition of Joldes, Muller and Popescu, "Tight and rigorous error bounds for basic
// building blocks of double-word arithmetic" (ACM TOMS 44, 2017), with both parts' errors carried
// (relative error below 3 u^2 with u = 2^-24).  The multiply-add of the translations is in owner.cu.
// Nothing here is reassociated (device code keeps IEEE order without fast-math), and there is no
// product that could be contracted into an FMA.
#pragma once
#include <cuda_runtime.h>
#include "fmm_common.cuh"

namespace fmm {

struct ff {
    float hi, lo;
    ff() = default;
    __host__ __device__ constexpr ff(float v) : hi(v), lo(0.f) {}
    __host__ __device__ constexpr ff(float h, float l) : hi(h), lo(l) {}
};

__device__ __forceinline__ void ff_two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

__device__ __forceinline__ void ff_fast_two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    e = b - (s - a);
}

__device__ __forceinline__ ff operator+(ff a, ff b)
{
    float s, e, t, f;
    ff_two_sum(a.hi, b.hi, s, e);
    ff_two_sum(a.lo, b.lo, t, f);
    e += t;
    ff_fast_two_sum(s, e, s, e);
    e += f;
    ff_fast_two_sum(s, e, s, e);
    return ff(s, e);
}

// nearest float-float to a double
__device__ __forceinline__ ff ff_from(double d)
{
    const float h = (float)d;
    return ff(h, (float)(d - (double)h));
}

} // namespace fmm
