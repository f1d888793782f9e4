// sph_divisor.cuh -- several correctly rounded FP64 quotients by one divisor.
// Plain C++ too (without FMA contraction), for the test on the CPU.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SPH_DIV_FN __device__ __forceinline__
#else
#define SPH_DIV_FN inline
#endif

namespace sph {

#ifdef __CUDACC__
SPH_DIV_FN double div_mul(double a, double b) { return __dmul_rn(a, b); }
SPH_DIV_FN double div_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
static __device__ __noinline__ double plain_quotient(double a, double b) { return a / b; }
#else
SPH_DIV_FN double div_mul(double a, double b) { return a * b; }
SPH_DIV_FN double div_fma(double a, double b, double c) { return std::fma(a, b, c); }
SPH_DIV_FN double plain_quotient(double a, double b) { return a / b; }
#endif

// Quotients a / b from r = RN(1 / b): q0 = RN(a r), the remainder a - b q0 by
// an FMA, and RN(q0 + r * remainder) -- Markstein's correction (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990).  A multiply and two FMAs for each quotient
// after the first division, instead of a division sequence (about ten FP64
// instructions and a branch).
//
// The published theorem asks for a q0 within one ulp of a / b and an exact
// remainder; RN(a r) may be 1.5 ulp off, and the remainder then rounded.  The
// result is the correctly rounded quotient all the same.  With a, b scaled to
// [1, 2), q = a / b, and errors in ulps of q:
//  - |b r - 1| <= b 2^-54, so |q0 - q| <= a/2 + 1/2 when a < b (q < 1) and
//    <= a/4 + 1/2 when a >= b.  The corrected value, before its last rounding,
//    differs from q by at most |q0 - q| |b r - 1|, plus 2^-52 / b for the
//    remainder's rounding, which happens only when |q0 - q| > 1: by less than
//    1.4 * 2^-52 in all.  It can be rounded to another number than q only when
//    a midpoint of two numbers lies nearer to q than that, so that |q0 - q| is
//    1/2 or 3/2 but for 1.4 * 2^-52.
//  - 3/2: then a / 2 >= 1 - 1.4 * 2^-52 and b > a, which only a = 2 - 2^-51,
//    b = 2 - 2^-52 meet, and their q lies next to a number.
//  - 1/2: the remainder is exact.  q differs from the midpoint by at least
//    g = 2^-53 / b, a quotient of 53-bit integers never being a midpoint, and
//    the corrected value from q by at most (1/2 + g) b 2^-54, which is less
//    than g as long as b b < 4 (1 - 2^-53): for every b.
// That holds while a, r and q0 lie away from the ends of the range.  A zero a
// with a finite r gives q0 = +-0, the quotient with its sign; every other
// operand takes the division itself, as a call: inlined, it was computed beside
// each quotient (k_finish executed 1,900 instructions a warp).
struct Divisor {
    double b, r;
    bool ok;
    SPH_DIV_FN explicit Divisor(double b_) : Divisor(b_, 1.0 / b_) {}
    SPH_DIV_FN Divisor(double b_, double r_) : b(b_), r(r_)
    {
        ok = fabs(r) > 0x1p-1000 && fabs(r) < 0x1p+1000;
    }
    SPH_DIV_FN double div(double a) const
    {
        const double q0 = div_mul(a, r);
        const double aq = fabs(q0);
        if (ok && aq > 0x1p-900 && aq < 0x1p+1000 && fabs(a) > 0x1p-900)
            return div_fma(div_fma(-q0, b, a), r, q0);
        if (ok && a == 0.0) return q0;
        return plain_quotient(a, b);
    }
};

}  // namespace sph
