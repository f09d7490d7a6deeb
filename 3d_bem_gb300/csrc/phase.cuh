// phase.cuh -- distances, and sine and cosine of small phase differences, shared by
// the FP64 kernels that take exp(ikr) as exp(ik r_c) exp(ik (r - r_c)).
#pragma once
#include <cuda_runtime.h>

namespace bemgpu {

// sqrt(x), x > 0, where ir = rsqrt(x) is needed anyway: one step of Newton's method
// for r^2 = x (Heron's rule r + (x / r - r) / 2, with 1 / r from ir) from r = x ir,
// the residual x - r^2 without rounding by an FMA. x ir is off by e of about 2e-16,
// the step leaves e^2 / 2 and its own rounding: half an ulp and 1e-31 of r.
__device__ __forceinline__ double newton_sqrt(double x, double ir) {
  const double r = x * ir;
  return fma(0.5 * ir, fma(-r, r, x), r);
}

// sin and cos of x, |x| <= X, by their Taylor series to x^(2 NS + 1) and
// x^(2 NC): for X = 0.35 (6, 6) the first terms left out are below 3e-19 and
// 5e-18 of the functions, for X = 1 (8, 9) below 1e-17 and 8e-19.
template <int NS, int NC>
__device__ __forceinline__ void sincos_taylor(double x, double& sn, double& cs) {
  constexpr double is[9] = {1.0,
                            -1.0 / 6,
                            1.0 / 120,
                            -1.0 / 5040,
                            1.0 / 362880,
                            -1.0 / 39916800,
                            1.0 / 6227020800.0,
                            -1.0 / 1307674368000.0,
                            1.0 / 355687428096000.0};
  constexpr double ic[10] = {1.0,
                             -1.0 / 2,
                             1.0 / 24,
                             -1.0 / 720,
                             1.0 / 40320,
                             -1.0 / 3628800,
                             1.0 / 479001600.0,
                             -1.0 / 87178291200.0,
                             1.0 / 20922789888000.0,
                             -1.0 / 6402373705728000.0};
  const double t = x * x;
  double ps = is[NS], pc = ic[NC];
#pragma unroll
  for (int q = NS - 1; q >= 1; q--) ps = fma(ps, t, is[q]);
#pragma unroll
  for (int q = NC - 1; q >= 0; q--) pc = fma(pc, t, ic[q]);
  sn = fma(x * t, ps, x);
  cs = pc;
}

}  // namespace bemgpu
