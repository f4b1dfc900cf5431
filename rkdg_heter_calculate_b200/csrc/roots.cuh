// FP64 reciprocal and square root of the flux arithmetic.
//
// The hardware's approximate seeds (PTX rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64, relative error about 2^-20) refined by one
// third-order Householder step each (A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970, ch. 4): with the seed's
// error e = 1 - x y (reciprocal) or e = 1 - x y^2 (root) the step keeps the
// series of 1/(1 - e) = 1 + e + e^2 and of (1 - e)^(-1/2) = 1 + e/2 + 3/8 e^2,
// so what is left, e^3 and 5/16 e^3, is below 2^-56, under the rounding of
// the last operation: within one unit in the last place of the exact value.
// Three (reciprocal) and six (root) FP64 operations without a branch, where
// the IEEE forms take about nine each and a slow-path test: the stage kernel
// makes some 40 of them per element and is bound by their chain.
// Arguments outside the normal range (zero or infinite density, say) give
// NaN, which the state check of a stage reports like any other.
#pragma once

namespace rkdg {

__device__ __forceinline__ double rcp_f64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// sqrt(x) and its reciprocal; 1e-300 keeps the seed finite at x = 0 (the
// root is then 0, its reciprocal some 1e150) and vanishes in the rounding of
// any argument above 1e-284.
__device__ __forceinline__ void roots_f64(double x, double& root, double& inv_root) {
    const double a = x + 1e-300;
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double h = e * fma(0.375, e, 0.5);
    root = fma(t, h, t);
    inv_root = fma(y, h, y);
}
__device__ __forceinline__ double sqrt_f64(double x) {
    double r, i;
    roots_f64(x, r, i);
    return r;
}

}  // namespace rkdg
