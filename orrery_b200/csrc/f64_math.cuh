// The softened inverse distance of the FP64 (bit-exact) paths: the correctly
// rounded reciprocal of the correctly rounded square root, as the reference's
// host code computes 1 / std::sqrt(x) (include/orrery/core/softening.hpp:83-100).
//
// Method. y0, the hardware's 20-bit estimate of x^-1/2, is refined by one
// cubic step of the Newton-Householder family (Householder, "The Numerical
// Treatment of a Single Nonlinear Equation", 1970): with e = 1 - x y0^2,
//   y = y0 + y0 e (1/2 + 3/8 e),   error (5/16) e^3,
// where y0^2 is exact (y0's low word is zero: 21 significant bits) and e is
// rounded once. |e| is at most 2^-19.03 (measured over every high word of [1, 4);
// y0 does not depend on the low word, so the ends of each decide), which makes the
// error of the cubic step 2^-58.7 relatively, and y, rounded, within 0.52 ulp of
// x^-1/2. Then two corrections in Markstein's form
// ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990), each one residual and one rounding:
//   g = x y,  s = g + (x - g^2) (y / 2)      the square root,
//   r = y + y (1 - s y)                      its reciprocal.
// Before their last rounding s and r are within 2^-103 of sqrt(x) and 1 / s
// relatively. Arguments whose root or reciprocal lies that near a midpoint of
// two doubles form a short list: the x with x 2^k = M^2 - j, and all x (up to
// three) whose rounded root is an s with s M = 2^k - j, for odd 54-bit M and small
// j. They are all that can round wrongly. The tests form the list and check every
// member, on the device and in exact arithmetic for every y within 0.52 ulp
// (test_direct_gpu.py, test_inverse_root_host.py). Only the root 2 - 2^-52 (times
// a power of two) fails, whose reciprocal can tie; its two arguments are left to
// the general operations. (With y off by 0.566 ulp others would fail too.)
//
// The FP64 pipe bounds the paths that use it: this takes 10 FP64 operations
// where the general square root and division took about 23 (a pair term 28
// instead of about 41).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ob {

// Arguments the short sequence covers: 2^-895 <= x < 2^897 (no intermediate
// result leaves the normal range), the low word below 2^32 - 2 (the two x whose
// root is 2 - 2^-52 are 4 - 2^-50 and 4 - 2^-51, times a power of four). The
// others -- zero, subnormal, huge, infinite, negative and NaN among them -- take
// the general operations.
__device__ __forceinline__ bool inverse_root_in_range(double x) {
    return static_cast<uint32_t>(__double2hiint(x) - 0x08000000) < 0x70000000u &&
           static_cast<uint32_t>(__double2loint(x)) < 0xfffffffeu;
}

__device__ __forceinline__ double inverse_root_in_range_rn(double x) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    const double e = __fma_rn(-x, __dmul_rn(y0, y0), 1.0);
    const double y = __fma_rn(__dmul_rn(y0, e), __fma_rn(e, 0.375, 0.5), y0);
    // y / 2 by its exponent (y is normal), off the FP64 pipe.
    const double half = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    const double g = __dmul_rn(x, y);
    const double s = __fma_rn(__fma_rn(-g, g, x), half, g);
    return __fma_rn(__fma_rn(-s, y, 1.0), y, y);
}

__device__ __forceinline__ double inverse_root_general(double x) {
    return __ddiv_rn(1.0, __dsqrt_rn(x));
}

__device__ __forceinline__ double inverse_root(double x) {
    return inverse_root_in_range(x) ? inverse_root_in_range_rn(x) : inverse_root_general(x);
}

} // namespace ob
