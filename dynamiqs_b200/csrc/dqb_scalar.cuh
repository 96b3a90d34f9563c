// FP64 scalar functions of the step control, in FP64 multiply-adds from an FP32 start.  No CUDA
// header is needed, so that a host compiler can test them (tests/test_scalar_functions.py).
#pragma once

namespace dqb {

// x / y, correctly rounded, for the error and starting-step norms (x >= 0): the reciprocal of y
// from FP32 by two Newton steps (within an ulp), then the quotient corrected by its residual
// (P. Markstein, IBM J. Res. Dev. 34, 1990).  The division where y lies outside 1e-30..1e30 or
// x beyond 1e270 (zero, infinite and NaN y and infinite x included).  x = 0 is exact; below
// 1e-270, where the residual underflows, the error can reach 1.5 ulp: a squared error of
// FP32 stages never lies there.  The division costs sparse-DIA n = 4096 solves 1.7%,
// n = 256 stencil solves 1.8% and sesolve 1%; the n <= 64 banded kernel is 1 to 3% faster with it.
__device__ __forceinline__ double ratio(double x, double y) {
  const float f = (float)y;
  if (f > 1e-30f && f < 1e30f && x < 1e270) {
    double r = (double)__frcp_rn(f);
    r = fma(r, fma(-y, r, 1.0), r);
    r = fma(r, fma(-y, r, 1.0), r);
    const double q = x * r;
    return fma(fma(-y, q, x), r, q);
  }
  return x / y;
}

// e^(-1/5) for e between 1e-30 and 1e30: an FP32 start (relative error below 1e-5) and two
// Newton steps x <- x + x (1 - e x^5) / 5, whose error is 3 times the square of the one
// before; at most 0.95 ulp from the exact value over the range (pow(e, -0.2) rounds the
// exponent too and is 7 ulp off at its ends).  pow otherwise.  The controller computes it once
// per step, alone, where pow's latency was 4% of a small instance's step.
__device__ __forceinline__ double inverse_fifth_root(double e) {
  const float f = (float)e;
  if (!(f > 1e-30f && f < 1e30f)) return pow(e, -0.2);
  double x = (double)exp2f(-0.2f * log2f(f));
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double x2 = x * x;
    x = fma(0.2 * x, fma(-e * x, x2 * x2, 1.0), x);
  }
  return x;
}

}  // namespace dqb
