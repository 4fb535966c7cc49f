// quotient.cuh -- correctly rounded FP64 quotients that share a divisor.
//
// The plain engine's results are those of IEEE divisions, one after another.
// A division on this GPU is a seed, Newton steps and a check that may call a
// slow path, some twenty instructions of which the reciprocal is the larger
// part, and it is repeated for every numerator.  Where several numerators
// have one divisor, the reciprocal is made once and each quotient takes four
// FP64 instructions, with the bits of the IEEE division:
//
//   P. W. Markstein, "Computation of elementary functions on the IBM RISC
//   System/6000 processor", IBM J. Res. Dev. 34 (1990): with y = RN(1/b) and
//   q a faithful rounding of a/b, r = a - b q is exact in one FMA and
//   RN(q + r y) = RN(a/b), when nothing over- or underflows.
#pragma once

#include "common.cuh"

namespace rtb {
namespace f64 {

// y = RN(1/b) and yl, the rest of 1/b to about 2^-105.
struct Divisor {
    double b, y, yl;
};

__device__ __forceinline__ Divisor divisor(double b) {
    const double y = __drcp_rn(b);
    return Divisor{b, y, fma(-b, y, 1.0) * y};
}

// RN(a / d.b), for a and b well inside the normal range, or a = +0: the
// double-word product a (y + yl) is within 0.5 + 2^-51 ulp of the quotient,
// hence faithful.
__device__ __forceinline__ double quot(double a, const Divisor& d) {
    const double q = fma(a, d.y, a * d.yl);
    const double r = fma(-d.b, q, a);
    return fma(r, d.y, q);
}

// RN(a / b) for b = 1 + e, |e| < 2^-28, and y = RN(1/b): a - a e is within
// 0.5 + 2^-3 ulp of the quotient (the next term is a e^2).
__device__ __forceinline__ double quot_by_unit(double a, double b, double e, double y) {
    const double q = fma(-a, e, a);
    const double r = fma(-b, q, a);
    return copysign(fma(r, y, q), a);
}

// 0 < |a| < 2^-900: residuals of its quotient could underflow.
__device__ __forceinline__ bool tiny(double a) {
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return hi < 0x07b00000u && (hi | (unsigned)__double2loint(a)) != 0u;
}

}  // namespace f64
}  // namespace rtb
