// f64_steps.cuh -- FP64 reciprocal root, root, quotient, sine and cosine from few instructions, for kernels that the
// FP64 pipe bounds (2 lanes a clock and SM).
//
// Root and quotient: the hardware's approximation (about 2^-20) improved by one third-order Householder step, in the form
// that the binomial and the geometric series give it (A. S. Householder, The Numerical Treatment of a Single
// Nonlinear Equation, 1970, ch. 4): with t = 1 - x y^2
//     x^(-1/2) = y (1 - t)^(-1/2) = y (1 + t/2 + 3 t^2/8 + ...),      t about 2^-19: the next term is 5/16 t^3 = 2^-58.7
// and with e = 1 - b y
//     1/b = y / (1 - e) = y (1 + e + e^2 + ...),                       e about 2^-20: 2^-60
// followed, for a quotient, by one residual correction q + y (a - b q).  Sine and cosine: the nearest of 256 angles from a
// table and the Taylor series about it (|d| <= pi/256: d^7/7! = 8e-18 is dropped).
// tests/test_f64_steps_gpu.py holds them against CUDA's functions.  Arguments: normal numbers whose results are
// normal (the approximations flush others to zero).
#pragma once
#include "common.cuh"

namespace mb {

__device__ __forceinline__ double rsqrt_step(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = fma(-(x * y), y, 1.0);
    return fma(t * y, fma(t, 0.375, 0.5), y);
}
__device__ __forceinline__ double sqrt_step(double x) { return x > 0.0 ? x * rsqrt_step(x) : sqrt(x); }
__device__ __forceinline__ double quotient_step(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

constexpr int kAngles = 256;

// table[i] = (sin, cos) of 2 pi i / 256, by the threads of a block (which then synchronises)
__device__ __forceinline__ void fill_angles(double2* table) {
    for (int i = threadIdx.x; i < kAngles; i += blockDim.x) {
        double s, c;
        sincospi(i * (2.0 / kAngles), &s, &c);
        table[i] = make_double2(s, c);
    }
}

// sin and cos of 2 pi turn x / 256
__device__ __forceinline__ void sincos_step(const double2* table, double x, double turn, double* s, double* c) {
    constexpr double kStep = 2.0 * kPi / kAngles;
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds
    const double z = fma(x, turn, kMagic);
    const double f = fma(x, turn, kMagic - z);
    const double2 t = table[__double2loint(z) & (kAngles - 1)];
    constexpr double k2 = kStep * kStep;
    const double q = f * f;
    const double sd = f * fma(q, fma(q, kStep * k2 * k2 / 120.0, -kStep * k2 / 6.0), kStep);
    const double cm = q * fma(q, fma(q, -k2 * k2 * k2 / 720.0, k2 * k2 / 24.0), -0.5 * k2);  // cos - 1
    *s = fma(t.y, sd, fma(t.x, cm, t.x));
    *c = fma(-t.x, sd, fma(t.y, cm, t.y));
}

}  // namespace mb
