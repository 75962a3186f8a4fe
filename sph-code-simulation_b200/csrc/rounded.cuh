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
//
// What the method gives: roots and reciprocals of an approximation within a unit
// in the last place are rounded, a reciprocal's divisor with a significand of all
// ones excepted (all_ones below); quotients need the rounded reciprocal.  Quick's
// div and div0 take one that is good to about an ulp: theirs are the rounded
// quotients but for operands whose quotient lies next to the middle of two doubles
// (2 in 10^8 of the nearest there are, none of 10^9 random ones), or a unit off
// for a divisor of all ones.  tests/cpp/rounded_ops.cu counts all of them against
// CUDA's operations.
#pragma once

namespace sphgpu {

// True when |x| is in [2^-300, 2^300]: no step below then overflows or loses
// bits to underflow.
__device__ __forceinline__ bool mid_range(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return hi - ((1023u - 300u) << 20) < (600u << 20);
}

// True for a significand of all ones, the one exception of the reciprocal's
// correction: 1 / b then lies just above the middle of a power of two and the
// next double, and a y of that power ties down to itself.
__device__ __forceinline__ bool all_ones(double x)
{
    return (unsigned)__double2loint(x) == 0xffffffffu && ((unsigned)__double2hiint(x) | 0xfff00000u) == 0xffffffffu;
}
// False for the few positive a (and others, one in 2^31) whose rounded root is a
// power of two less one unit in the last place, a significand of all ones.
__device__ __forceinline__ bool root_not_ones(double a) { return (unsigned)__double2loint(a) < 0xfffffffeu; }

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

// 1 / b, rounded, from a y a few units off (corrected twice) and for a significand
// of all ones too: the double after the power of two
__device__ __forceinline__ double recip_any(double b, double y)
{
    const double r = recip_rn(b, recip_rn(b, y));
    return __hiloint2double(__double2hiint(r), __double2loint(r) | (all_ones(b) ? 1 : 0));
}

// a / b, rounded, from y = 1 / b rounded
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// Quotients and roots of one pair: Quick takes the forms above and notes when a
// result may have left the range where they hold (its pair is then computed
// again with Ieee); no branch in between, so independent operations overlap.
// A result in 2^-400 .. 2^400 then holds as above: an operand outside the
// exponent range yields zero, infinity or NaN.  (Operands below 2^-900 with such a
// quotient are not flagged: their residual may lose bits, and the result its
// last.)
struct Ieee {
    static constexpr bool quick = false;
    bool bad = false;
    __device__ __forceinline__ double inverse(double b) { return 1.0 / b; }
    __device__ __forceinline__ double over(double a, double b, double) { return a / b; }
    __device__ __forceinline__ double div(double a, double b) { return a / b; }
    __device__ __forceinline__ double div0(double a, double b) { return a / b; }
    __device__ __forceinline__ double root(double a) { return sqrt(a); }
    __device__ __forceinline__ double root0(double a) { return sqrt(a); }
};
struct Quick {
    static constexpr bool quick = true;
    bool bad = false;
    __device__ __forceinline__ double check(double q)
    {
        const unsigned hi = (unsigned)__double2hiint(q) & 0x7fffffffu;
        bad = bad || hi - ((1023u - 400u) << 20) >= (800u << 20);
        return q;
    }
    // 1 / b to about an ulp, for over()
    __device__ __forceinline__ double near(double b)
    {
        const double y = rcp_seed(b);
        const double e = __fma_rn(-b, y, 1.0);
        return __fma_rn(y, __fma_rn(e, e, e), y);
    }
    // 1 / b
    __device__ __forceinline__ double inverse(double b) { return check(recip_rn(b)); }
    // a / b with y = 1 / b taken before; a may be zero
    __device__ __forceinline__ double over(double a, double b, double y)
    {
        const double q = quot_rn(a, b, y);
        if(a != 0.0) check(q);
        return q;
    }
    __device__ __forceinline__ double div(double a, double b) { return check(quot_rn(a, b, near(b))); }
    // a / b, a may be zero
    __device__ __forceinline__ double div0(double a, double b)
    {
        const double y = near(b);
        check(y);
        return over(a, b, y);
    }
    __device__ __forceinline__ double root(double a) { return check(root_rn(a, rsqrt_near(a))); }
    // sqrt(a), a may be zero
    __device__ __forceinline__ double root0(double a) { return a > 0.0 ? root(a) : (check(a == 0.0 ? 1.0 : 0.0), 0.0); }
};

}  // namespace sphgpu
