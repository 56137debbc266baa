// recip.cuh -- reciprocal of a double.
#pragma once

namespace olamgpu {

// Out of line: with the division inside it the loop of the column solve keeps
// more registers (k_wrt_begs at NXP=100, 60 levels 328 us a stage against 326,
// at NXP=50, 30 levels 58 against 55).
static __device__ __noinline__ double quotient(double x) { return 1.0 / x; }

// 1 / x by Newton-Raphson, y <- y + y (1 - x y), from the instruction set's
// approximate reciprocal (20 bits): each step squares the relative error, so
// two leave the last rounding, and the result is within 1 ulp of the
// quotient's.  Where the iteration does not give a nonzero number (x zero,
// infinite, NaN or subnormal, or 1 / x subnormal) the division does.  The
// division throughout: 351 and 54 us.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  y = fma(y, fma(-x, y, 1.0), y);
  if (!(fabs(y) > 0.0)) y = quotient(x);
  return y;
}

}  // namespace olamgpu
