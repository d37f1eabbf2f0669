// rt_fast_math.h -- FP64 reciprocal and square root for the step loops, host/device.
//
// The tracers' arguments (r^2 and r^6 of a point) are far from the ends of the range,
// so these forms leave special arguments out and are one straight line of fused
// operations.  Measured with 1.0 / v and sqrt(v) / with these: 2048^2 FP64 33.05 / 31.11 ms,
// 512^2 FP64 2.52 / 2.36, 1024^2 Kerr-Newman 22.0 / 21.5, a 640x360 frame with the torus
// 14.6 / 13.6.
//
// Both start from the hardware's approximation (PTX rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64, about 20 bits) and refine it by the convergent products of
// R. E. Goldschmidt ("Applications of division by convergence", M.Sc. thesis, MIT 1964),
// in fused operations as in P. Markstein, "Software division and square root using
// Goldschmidt's algorithms" (6th Conference on Real Numbers and Computers, 2004).  The
// last step of each is Markstein's correction by a fused residual ("Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990), which rounds correctly: the results are those of 1.0 / v and sqrt(v), but for a
// reciprocal whose argument has a significand of all ones, which is one ulp low.
//
// That holds for arguments in [2^-900, 2^1020].  For zero, subnormal, negative (the
// root) and infinite arguments and NaN the result is NaN: the seed is infinite, zero or
// NaN, and the steps multiply infinity by zero or subtract infinities.  Other arguments
// have no such mark: below 2^-900 a root may be an ulp off, and from 2^1022 on the
// reciprocal's seed is flushed to zero and the result is 0.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define RT_FM_FN __host__ __device__ __forceinline__
#else
#define RT_FM_FN inline
#endif

namespace relsim {

// 1 / v from a seed y of at least 18 bits.  With e = 1 - v y, 1 / v = y / (1 - e) =
// y (1 + e)(1 + e^2)(1 + e^4)...: two factors leave a relative error of e^4 = 2^-72 and
// two roundings, in all an ulp.  The square is formed beside the first product, so that
// the chain is one operation shorter than by two Newton-Raphson steps (2048^2 FP64
// 31.36 / 31.28 ms, 1024^2 Kerr-Newman 21.64 / 21.57).
// The correction y + y (1 - v y) then errs by (1 / v) (1 - v y)^2 before it rounds,
// always to the low side.  With b in [1, 2) for v, y off by an ulp of 1 / b, 2^-53, at
// most and a midpoint m of two neighbours of 1 / b, it can only round to the wrong side
// if 0 < 1 / b - m < b 2^-106, that is, for the 53-bit integer B of b and the odd 54-bit
// integer M of m, if B M = 2^106 - j with 0 < j < b^2 <= 4.  Factorised, these three numbers
// leave j = 1 with B = 2^53 - 1 (all ones) and j = 2 with 32 significands, of which those
// with b^2 > 2 need a y off by sqrt(2) / b ulp or more; the tests run all 32.  (e^4 adds
// 2^-18 of an ulp, which would let in j = 4 with b within 2^-17 of 2; there is none.)
RT_FM_FN double refine_rcp(double v, double y) {
    const double e = fma(-v, y, 1.0);
    y = fma(y, e, y);
    y = fma(y, e * e, y);
    return fma(y, fma(-v, y, 1.0), y);
}

// sqrt(v) from a seed y of 1 / sqrt(v) of at least 18 bits.  g = v y goes to sqrt(v) and
// h = y / 2 to 1 / (2 sqrt(v)): with r = 1/2 - g h, where 2 g h = 1 - 2 r, both are short
// of their limits by the factor (1 - 2 r)^(1/2) = 1 - r - ..., so g + g r and h + h r
// leave an error of the order of r^2: 2^-35 and 2^-69.  The correction adds the residual
// v - g^2 divided by 2 g.  h is left within two ulp of 1 / (2 sqrt(v)).
RT_FM_FN double refine_sqrt(double v, double y, double& h) {
    double g = v * y;
    h = 0.5 * y;
    double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, v), h, g);
}

RT_FM_FN double refine_sqrt(double v, double y) {
    double h;
    return refine_sqrt(v, y, h);
}

// On the host, which has no such seeds, the operations themselves.
RT_FM_FN double fast_rcp(double v) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    return refine_rcp(v, y);
#else
    return 1.0 / v;
#endif
}

// sqrt(v), and 1 / (2 sqrt(v)) within two ulp from the same steps.
RT_FM_FN double fast_sqrt(double v, double& half_inverse) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    return refine_sqrt(v, y, half_inverse);
#else
    const double root = std::sqrt(v);
    half_inverse = 0.5 / root;
    return root;
#endif
}

RT_FM_FN double fast_sqrt(double v) {
    double half_inverse;
    return fast_sqrt(v, half_inverse);
}

}  // namespace relsim
