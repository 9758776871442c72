// Correctly rounded FP64 quotients without a division each.
#pragma once

namespace stitch::b200 {

// a / b correctly rounded from y = 1 / b correctly rounded (Markstein's
// quotient correction: with q within one unit in the last place of a / b and r
// = a - b q, RN(q + r y) is RN(a / b)). RN(a y) can be 1.5 units off, so one
// correction first makes q faithful (its remainder may round, far below a
// unit); the second has an exact remainder. Needs quotient and remainders
// clear of overflow and underflow. Three such quotients over one reciprocal
// cost a division and 15 operations instead of three divisions of some 36
// issue slots each, the FP64 pipe being what bounds this kernel.
__device__ __forceinline__ double quotient(double a, double b, double y) {
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// v / 255 correctly rounded for 0 and for normal v: RN(1 / 255) is within
// 2^-56 of 1 / 255 relatively, so RN(v y) is within 0.75 units of v / 255 and
// one correction is enough.
__device__ __forceinline__ double over255(double v) {
    constexpr double y = 1.0 / 255.0;
    const double q = __dmul_rn(v, y);
    return __fma_rn(__fma_rn(-255.0, q, v), y, q);
}

// Whether quotient(a, b, y) stays clear of overflow and underflow: both
// magnitudes within 2^-400 .. 2^400, or a zero (tests of the exponents).
__device__ __forceinline__ bool quotient_range(double a, double b) {
    const unsigned x = static_cast<unsigned>(__double2hiint(a)) & 0x7fffffffu, z = static_cast<unsigned>(__double2hiint(b)) & 0x7fffffffu;
    constexpr unsigned lo = (1023u - 400u) << 20, span = 800u << 20;
    return z - lo < span && (x - lo < span || (x | static_cast<unsigned>(__double2loint(a))) == 0u);
}

}  // namespace stitch::b200
