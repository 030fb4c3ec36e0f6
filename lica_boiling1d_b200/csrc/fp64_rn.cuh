// Correctly rounded FP64 reciprocals and quotients without a branch.
//
// `a / b` and `1.0 / b` carry a test for extreme operands and a call behind it, so two
// independent divisions of one thread do not overlap: measured on a B200, 64 cycles for 1/b,
// 115 for a/b, and 123 for two independent 1/b.  These forms are straight-line FMA chains
// that do overlap, and the test for extreme operands (`ordinary`) is apart, to be made once
// for a group of divisions; where it fails the caller takes the plain operator.  The results
// are the IEEE quotients bit for bit.
//
// Method: the reciprocal by a cubic step from the hardware's 20-bit seed, to within a unit
// in the last place, then Markstein's correction, whose result is the correctly rounded 1/b
// for every b but a mantissa of all ones; the quotient by Markstein's correction of a
// quotient within a unit in the last place (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  A first
// correction brings a * (1/b), up to 1.5 units off, to within one.
#pragma once

namespace lica {
namespace rn {

// exponent of b within 2^-400 .. 2^400, and not a mantissa of all ones
__device__ __forceinline__ bool ordinary(double b) {
    const int hi = __double2hiint(b), lo = __double2loint(b);
    const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
    return (e - 623u) <= 800u && !((hi & 0xfffff) == 0xfffff && lo == -1);
}

__device__ __forceinline__ double recip(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    e = __fma_rn(e, e, e);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, e, y);
}

// a / b given y = recip(b); a and b ordinary
__device__ __forceinline__ double quot(double a, double b, double y) {
    double q = a * y;
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

}  // namespace rn
}  // namespace lica
