// rounded.cuh — correctly rounded FP64 roots and quotients without the
// special-case branches of the general operations, for operands known to lie
// in the middle of the exponent range.
//
// Markstein's final-correction method (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1), 1990): an approximation good to about an ulp, its exact
// residual by a fused multiply-add, and one fused correction round as the
// exact quotient, reciprocal or root does.  The seeds are the hardware's
// double-precision approximations (about 2^-20), refined by one third-order
// step of the Taylor series of 1 / sqrt(1 - e) and 1 / (1 - e).  The fused
// operations are explicit, so the files built without contraction keep every
// other operation as written.
#pragma once

namespace sphgpu {

// True when |x| is in [2^-300, 2^300]: no step below then overflows or loses
// bits to underflow.
__device__ __forceinline__ bool mid_range(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return hi - ((1023u - 300u) << 20) < (600u << 20);
}

__device__ __forceinline__ double rsqrt_seed(double a)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}

__device__ __forceinline__ double rcp_seed(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}

// 1 / sqrt(a) to about an ulp: y (1 + e / 2 + 3 e^2 / 8), e = 1 - a y^2
__device__ __forceinline__ double rsqrt_near(double a)
{
    const double y = rsqrt_seed(a);
    const double e = __fma_rn(-__dmul_rn(a, y), y, 1.0);
    return __fma_rn(__dmul_rn(y, e), __fma_rn(e, 0.375, 0.5), y);
}

// sqrt(a), rounded, from y ~ 1 / sqrt(a)
__device__ __forceinline__ double root_rn(double a, double y)
{
    const double s = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-s, s, a), __dmul_rn(0.5, y), s);
}

// 1 / b, rounded, from y ~ 1 / b
__device__ __forceinline__ double recip_rn(double b, double y) { return __fma_rn(__fma_rn(-b, y, 1.0), y, y); }

// 1 / b, rounded: y (1 + e + e^2), e = 1 - b y, then the correction
__device__ __forceinline__ double recip_rn(double b)
{
    const double y = rcp_seed(b);
    const double e = __fma_rn(-b, y, 1.0);
    return recip_rn(b, __fma_rn(y, __fma_rn(e, e, e), y));
}

// a / b, rounded, from y = 1 / b rounded
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

}  // namespace sphgpu
