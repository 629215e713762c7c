// 1/x for 1e-30 <= x <= 1e30: the hardware's approximation r, refined by Newton's iteration r <- r + r (1 - x r)
// without the special cases of a correctly rounded reciprocal, whose branches would keep the TVD faces of
// a level from being interleaved.
//
// Error: an iteration squares the relative error e of r and adds half a unit of the last place for its own
// rounding (the residual 1 - x r is one fused multiply-add, so that its rounding is e times smaller still).
// With e <= 2^-14 two iterations leave 2^-56 in FP64, and with the 2^-22 of the FP32 approximation one leaves
// 2^-44: the result is one of the two neighbours of 1/x, at most one unit from the correctly rounded
// value.  tests/test_gpu_reciprocal.py compares it with 1.0 / x over the range.
#pragma once

namespace mgpu {

__device__ __forceinline__ double rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}
__device__ __forceinline__ float rcp_newton(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(r, fmaf(-x, r, 1.0f), r);
}

}  // namespace mgpu
