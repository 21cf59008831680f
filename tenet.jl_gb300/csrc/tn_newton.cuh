// Reciprocals and roots in the chains of the FP64 factorisations: the hardware's approximations
// (some 20 bits) refined by Newton's iteration.
#pragma once

#include <cuda_runtime.h>

// 1/x of a positive x of [1e-290, 1e290]: two Newton–Raphson steps y ← y + y(1 − x·y), each of which
// doubles the correct bits
__device__ __forceinline__ double newton_reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
// √x of an x of [1e-290, 1e290]: one step of Goldschmidt's coupled iteration, g → √x and
// h → 1/(2√x) by r = 1/2 − g·h, then one Newton (Heron) step from the residual, g + (x − g²)·h
__device__ __forceinline__ double newton_root(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = x * y, h = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));  // y/2
  const double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  return fma(fma(-g, g, x), h, g);
}
