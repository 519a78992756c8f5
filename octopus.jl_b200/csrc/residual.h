// Quotients and square roots by residual correction, for divisors that are constant or shared (Markstein's method: P.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990)
// 111-119): an approximation from the shared reciprocal, its residual in one fused multiply-add, and one correction.
//
// With a reciprocal within three units in the last place, as every caller's is, the results are within one unit of the
// rounded quotient and root.  Host-compilable: the tests check that over random and extreme operands.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define OCTO_RESIDUAL __host__ __device__ __forceinline__
#else
#define OCTO_RESIDUAL inline
#endif

namespace octo {

// x / d, d not subnormal and rd its reciprocal; a zero comes without its sign.  Where the residual is not finite (a
// product that overflows, an infinite or NaN operand, d = 0) the product is the quotient.  For |x| < 2^-960 the residual
// can underflow, which leaves the product: seven units.
OCTO_RESIDUAL double quotient(double x, double d, double rd) {
    const double q = x * rd, r = fma(-q, d, x);
    return fabs(r) <= 1.7976931348623157e308 ? fma(r, rd, q) : q;
}

// The same of finite operands whose quotient does not overflow.
OCTO_RESIDUAL double quotient_in_range(double x, double d, double rd) {
    const double q = x * rd;
    return fma(fma(-q, d, x), rd, q);
}

// sqrt(v), v a positive normal number and rs the reciprocal of its root.
OCTO_RESIDUAL double root(double v, double rs) {
    const double s = v * rs;
    return fma(fma(-s, s, v), 0.5 * rs, s);
}

}  // namespace octo
