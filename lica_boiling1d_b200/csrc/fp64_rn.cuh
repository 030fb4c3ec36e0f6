// Correctly rounded FP64 reciprocals, quotients and square roots without a branch.
//
// Two independent divisions of one thread do not overlap when they are written with the
// operators: measured on a B200, 64 cycles for 1/b, 115 for a/b, and 123 for two independent 1/b.
// These forms are straight-line FMA chains that do overlap, and the test for extreme operands
// (`ordinary`) is apart, to be made once for a group of divisions; where it fails the caller
// takes the plain operator.  The results are the IEEE quotients bit for bit.
//
// Method: the reciprocal by a cubic step from the hardware's 20-bit seed, to within a unit
// in the last place, then Markstein's correction, whose result is the correctly rounded 1/b
// for every b but a mantissa of all ones; the quotient by Markstein's correction of a
// quotient within a unit in the last place (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  A first
// correction brings a * (1/b), up to 1.5 units off, to within one.  The square root by two
// coupled Newton steps (Goldschmidt) from the hardware's seed and a last correction, the
// rounding then checked by the remainder's size (Tuckerman's test): g is the rounded root of x
// exactly if -g ulp(g) < x - g^2 <= g ulp(g).
#pragma once

namespace lica {
namespace rn {

// |b| within 2^-400 .. 2^400
__device__ __forceinline__ bool in_range(double b) {
    return ((unsigned)__double2hiint(b) & 0x7fffffffu) - 0x26f00000u < 0x32000000u;
}
// and its mantissa not all ones
__device__ __forceinline__ bool ordinary(double b) {
    return in_range(b) && !(__double2loint(b) == -1 && (__double2hiint(b) & 0xfffff) == 0xfffff);
}

// ordinary, and a little less: without a branch, for the inside of a chain
__device__ __forceinline__ bool plain(double b) { return in_range(b) & (__double2loint(b) != -1); }

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

// sqrt(x), x in range (the test of the rounding needs nothing of the mantissa); ok is cleared where
// the result is not the correctly rounded root
__device__ __forceinline__ double root(double x, bool& ok) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    double r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    g = __fma_rn(__fma_rn(-g, g, x), h, g);
    // ulp(g) = 2^(exponent - 52): g >= 2^-200 here
    const double gu = g * __hiloint2double((__double2hiint(g) & 0x7ff00000) - (52 << 20), 0);
    const double rem = __fma_rn(-g, g, x);
    ok = ok && rem > -gu && rem <= gu;
    return g;
}

}  // namespace rn
}  // namespace lica
