// sum2.cuh — sums kept in two FP32 words s + c, c the rounding errors of s
// (Knuth's two-sum and Dekker's product error by FMA): close to FP64 accuracy at
// FP32 issue rates, where FP64 runs at two lanes a clock and SM.  The operations
// are written as single roundings; host code needs -ffp-contract=off.
#pragma once
#include <cmath>

#if defined(__CUDACC__)
#define SUM2_HD __host__ __device__ __forceinline__
#else
#define SUM2_HD inline
#endif

SUM2_HD float sum2_radd(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}

SUM2_HD float sum2_rmul(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}

// s + c += v
SUM2_HD void sum2_add(float &s, float &c, float v)
{
    const float z = sum2_radd(s, v), w = sum2_radd(z, -s);
    c = sum2_radd(c, sum2_radd(sum2_radd(s, -sum2_radd(z, -w)), sum2_radd(v, -w)));
    s = z;
}

// s + c += (h + l) t
SUM2_HD void sum2_mul_add(float &s, float &c, float h, float l, float t)
{
    const float p = sum2_rmul(h, t), e = fmaf(h, t, -p);
    sum2_add(s, c, p);
    c = sum2_radd(c, fmaf(l, t, e));
}

// sqrt(h + l) rounded to FP32, h > 0 the value's FP32 head
SUM2_HD float sum2_sqrt(float h, float l)
{
    const float r = sqrtf(h);
    return r + 0.5f * (fmaf(-r, r, h) + l) / r;
}
