// FP64 inverse distances for the pair kernels.
//
// The FP64 pair loops are bound by the FP64 pipe (64 lanes per SM), and a full
// library reciprocal square root plus its cube took about half of a pair's
// slots there: 82.6 ms for the 6.9e10 directed pairs of a 262,144-body
// evaluation is 22 FP64 instructions a pair. Here r^-3 (or r^-1) comes from the
// hardware's approximate reciprocal square root and one third-order step of the
// binomial series of (1 - e)^(-3/2) (or (1 - e)^(-1/2)) in the residual
// e = 1 - r^2 y^2:
//   r^-1 = y   (1 + e/2   + 3/8  e^2 + O(e^3))
//   r^-3 = y^3 (1 + 3/2 e + 15/8 e^2 + O(e^3))
// 6 FP64 operations for r^-3. The approximation's low word is zero, so y^2 is
// exact and e carries one rounding; the omitted terms stay below the result's
// rounding (the tests bound the whole error against extended precision). Very small,
// very large, zero and NaN arguments (outside [1e-200, 1e200]) are recognised
// by an integer test of the high word and take the library function.
#pragma once

#include <cuda_runtime.h>

__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// x within [2^-664, 2^664): the series step neither over- nor underflows.
__device__ __forceinline__ bool r2_ordinary(double x) {
    return (unsigned)(__double2hiint(x) - 0x16700000) < 0x53000000u;
}

// x^(-3/2) of an ordinary x
__device__ __forceinline__ double inv_r3_fast(double x) {
    const double y = rsqrt_seed(x), y2 = y * y;
    const double e = fma(-x, y2, 1.0);
    const double y3 = y2 * y;
    return fma(y3 * e, fma(1.875, e, 1.5), y3);
}

// x^(-1/2) of an ordinary x
__device__ __forceinline__ double inv_r_fast(double x) {
    const double y = rsqrt_seed(x), y2 = y * y;
    const double e = fma(-x, y2, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// x^(-1/2) of any x; 0 for x = 0 (a body and itself) and for NaN
__device__ __forceinline__ double inv_r_any(double x) { return x > 0.0 ? rsqrt(x) : 0.0; }

__device__ __forceinline__ double inv_r(double x) {
    double y = inv_r_fast(x);
    if (!r2_ordinary(x)) y = inv_r_any(x);
    return y;
}

// inv_r where x = 0 is common (a body among its own sources): no branch for it
__device__ __forceinline__ double inv_r_or_0(double x) {
    const bool zero = (__double2hiint(x) | __double2loint(x)) == 0;
    double y = inv_r_fast(x);
    if (!r2_ordinary(x) && !zero) y = inv_r_any(x);
    return zero ? 0.0 : y;
}

// m x^(-3/2), 0 for x = 0; the mass first where r^-3 alone may leave the range
__device__ __forceinline__ double m_inv_r3(double m, double x) {
    double s = m * inv_r3_fast(x);
    if (!r2_ordinary(x)) {
        const double v = inv_r_any(x);
        s = m * v * (v * v);
    }
    return s;
}
