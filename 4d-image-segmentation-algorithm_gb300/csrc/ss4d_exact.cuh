// ss4d_exact.cuh — the exactly rounded division by a constant of the kernels
// that keep the reference's FP64 rounding (units compiled with --fmad=false).
#pragma once

#include "ss4d_common.cuh"

namespace ss4d {

// x / d, rounded to nearest, for a divisor d > 0 known in advance with
// y = 1/d rounded to nearest (y == 0: no fast path).  A quotient from the
// reciprocal and one remainder correction (Markstein's iteration), then an
// exact acceptance test: the remainder x - q d (one FMA, correctly rounded) must
// be below d times half the spacing from q to its nearer neighbour; since
// that bound is a power-of-two multiple of d, hence exact, and rounding is
// monotonic, passing it proves q is the double nearest to x / d.  Otherwise
// (near a tie, zero, q outside [2^-400, 2^601)) the IEEE division decides.
__device__ __forceinline__ double div_by_const(double x, double d, double y)
{
    if (y != 0.0) {
        if ((__double_as_longlong(x) & 0x7fffffffffffffffLL) == 0)
            return x; // +-0 / d (a thresholded image is mostly zeros)
        const double q0 = x * y;
        const double q = fma(fma(-q0, d, x), y, q0);
        const long long b = __double_as_longlong(q);
        const int E = (int)((b >> 52) & 0x7ff) - 1023;
        if (E >= -400 && E <= 600) {
            const int e = E - 53 - ((b & 0xfffffffffffffLL) == 0 ? 1 : 0); // half spacing 2^e
            // d 2^e (a normal number: d in [2^-300, 2^300]) by adding e to d's
            // exponent, and |r| < d 2^e compared as the bit patterns of two
            // non-negative doubles: integer work only
            const long long lim = __double_as_longlong(d) + ((long long)e << 52);
            if ((__double_as_longlong(fma(-q, d, x)) & 0x7fffffffffffffffLL) < lim)
                return q;
        }
    }
    return x / d;
}

// reciprocal for div_by_const, or 0 where the divisor is outside the range
// its test needs (d in [2^-300, 2^300])
inline double div_const_recip(double d)
{
    return (d >= 0x1p-300 && d <= 0x1p300) ? 1.0 / d : 0.0;
}

} // namespace ss4d
