// hb_fastmath.cuh -- FP64 reciprocal and reciprocal square root from the
// hardware approximations, for the stage sets that do not need IEEE-rounded
// division and square root (the mixed-precision and the FMA FP64 sets).
#pragma once

#include <cuda_runtime.h>

namespace hb {

// Reciprocal and reciprocal square root in FP64: the hardware approximation
// (PTX rcp.approx.ftz.f64 / rsqrt.approx.ftz.f64) refined by two
// Newton-Raphson steps, each of which doubles the number of correct bits, to
// the FP64 rounding level.  Inputs are positive normal numbers (every
// divisor and radicand of a valid state is).
__device__ __forceinline__ double rcp64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

__device__ __forceinline__ double rsqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double h = 0.5 * y;
    double r = fma(-(x * y), h, 0.5);  // 1/2 - x y^2 / 2
    y = fma(y, r, y);
    h = 0.5 * y;
    r = fma(-(x * y), h, 0.5);
    return fma(y, r, y);
}

// The reciprocal square root by one step of fourth order from the approximation:
// with e = 1 - x y^2 it is y (1 + e/2 + 3 e^2 / 8 + 5 e^3 / 16) up to 35 e^4 / 128.
// For an approximation within 2^-19 of the root (e below 2^-18) that is below
// 2^-73.  6 operations, where two Newton-Raphson steps take 8; the last bit may
// differ, so the mixed set, whose FP32 stages would carry a flipped bit on, keeps
// the former.  One term less (and the reciprocal likewise, 3 operations for 4)
// leaves a bias of up to 2^-55 and was 2% faster a sweep, but after 100-200 steps of four blasts (250x125
// to 2048^2) the FMA tier's density was 2.8e-16 from the bit-exact path, geometric
// mean of the relative 2-norms, against 2.2e-16 with two Newton-Raphson steps for
// both and 2.0e-16 so.
__device__ __forceinline__ double rsqrt64_quartic(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(fma(0.3125, e, 0.375), e, 0.5), y);
}

}  // namespace hb
