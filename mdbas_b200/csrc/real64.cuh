// real64.cuh -- FP64 building blocks of the real-space pair kernels: 1/sqrt
// and 1/x by Newton steps and the scaled complementary error function.
//
// The pair kernels are bound by the FP64 pipe.  sqrt, three divisions, erfc and
// exp of the C library forms cost about 250 FP64 instructions per pair; the
// forms here about 60.  A pair's energy and force are within 6 x 2^-53 of exact
// (1.4 rms; tests/test_gpu_pair_functions.py); the forces of eight 3,000-atom
// boxes of water are 2.76e-15 from long double sums (with the library's
// functions 2.86e-15), their energies 2.3e-10 internal units (3.5e-10).  They
// hold on the range that the callers check; pairs outside it take the library
// forms.
#pragma once

#include "common.cuh"

namespace mdbas {

// 1/sqrt(x), x > 0 normal: the hardware's starting value (relative error
// below 2^-20) and one third-order Newton step (y (1 + e/2 + 3 e^2/8),
// e = 1 - x y^2), which leaves the rounding of the last operations.
__device__ __forceinline__ double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// sqrt(x) from y = rsqrt64(x): one Newton correction of x y.
__device__ __forceinline__ double sqrt64(double x, double y) {
  const double r = x * y;
  return fma(0.5 * y, fma(-r, r, x), r);
}

// 1/x, x > 0 normal: starting value and one third-order step.
__device__ __forceinline__ double rcp64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y * e, 1.0 + e, y);
}

// Coefficients in constant memory: an FP64 operation takes such an operand
// directly, where a 64-bit immediate costs two moves.
__constant__ static const double kErfcxC[19] = {
    1.0740069070883398, -0.8833944531698831, 0.5902283571040964,
    -0.31046726190066504, 0.11952776128767394, -0.026827234618821024,
    -0.001212416632445897, 0.003034061857623385, -0.0005483098232609487,
    -0.00027677618791188636, 0.00010756548241527724, 3.0392027377246628e-05,
    -1.7504489289456764e-05, -4.7770821878695634e-06, 2.839965105053344e-06,
    1.194847930350894e-06, -2.4033472884214317e-07, -2.2611900751571806e-07,
    -3.999345065213784e-08};
__constant__ static const double kExpC[12] = {  // 1 / k!, k = 2..13
    0.5, 0.16666666666666666, 0.041666666666666664, 0.008333333333333333,
    0.001388888888888889, 0.0001984126984126984, 2.48015873015873e-05, 2.7557319223985893e-06,
    2.755731922398589e-07, 2.505210838544172e-08, 2.08767569878681e-09, 1.6059043836821613e-10};

// erfc(x) exp(x^2) on [0, 6]: (x + 3) erfcx(x) is a polynomial of degree 18 in
// (x - 3) / (x + 3) to a relative 1.9e-17 (fit_erfc.py: Chebyshev
// interpolation in 70-digit arithmetic).  The map is that of M. M. Shepherd and
// J. G. Laframboise, Math. Comp. 36 (1981) 249, who take it over [0, inf).
constexpr double kErfcxMax = 6.0;
__device__ __forceinline__ double erfcx64(double x) {
  const double inv = rcp64(x + 3.0);
  const double t = (x - 3.0) * inv;
  double p = kErfcxC[18];
#pragma unroll
  for (int k = 17; k >= 0; --k) p = fma(p, t, kErfcxC[k]);
  return p * inv;
}

// exp(-u), 0 <= u <= 700: e^f 2^n with n the nearest integer to -u / ln 2 and
// ln 2 in two parts (n times the first is exact), e^f by its Taylor series
// (|f| <= 0.35: the first term left out is 4e-18).
__device__ __forceinline__ double expm64(double u) {
  const double big = 6755399441055744.0;  // 1.5 2^52: the sum rounds to an integer
  const double m = fma(u, -1.4426950408889634, big);
  const double n = m - big;
  double f = fma(n, -0.6931471805582987, -u);
  f = fma(n, -1.6465949582897082e-12, f);
  double p = kExpC[11];
#pragma unroll
  for (int k = 10; k >= 0; --k) p = fma(p, f, kExpC[k]);
  p = fma(f * f, p, f) + 1.0;
  return __hiloint2double(__double2hiint(p) + (__double2loint(m) << 20), __double2loint(p));
}

// exp(-(a2 + a2lo) r2) from a product in two parts (a2 + a2lo is alpha^2 to
// twice the precision): a rounded x^2 would put an error of x^2 ulps on it.
// a2lo r2 is less than half an ulp of u: it is added to what u's rounding left
// out, not to u.
__device__ __forceinline__ double expm64_product(double a2, double a2lo, double r2) {
  const double u = a2 * r2;
  const double g = expm64(u);
  return fma(-g, fma(a2lo, r2, fma(a2, r2, -u)), g);
}

// 2 alpha / sqrt(pi), alpha^2 in two parts, and the switch's factor and
// constant term.
struct EwaldConst {
  double g0, a2, a2lo, sw2, swc;
  __device__ __forceinline__ explicit EwaldConst(const PairParams &p)
      : g0(2.0 * p.alpha / kSqrtPi), a2(p.alpha * p.alpha), a2lo(fma(p.alpha, p.alpha, -a2)),
        sw2(p.switch2), swc(p.cutOff2 - 3. * p.cutOn2) {}
};

}  // namespace mdbas
