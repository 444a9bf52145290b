// pivot_rcp.cuh -- the reciprocal on the pivot chain of the banded elimination (topopt.cu).
#pragma once

namespace tptfem {

// Pivots whose reciprocal td_rcp holds: its approximation takes subnormals for zero and
// gives none.
constexpr double TD_PIVOT_MIN = 0x1p-1021, TD_PIVOT_MAX = 0x1p1021;

// 1 / x, x in [TD_PIVOT_MIN, TD_PIVOT_MAX], by Newton-Raphson from the hardware's
// approximate reciprocal (rcp.approx.ftz.f64, PTX ISA: relative error below 2^-20): two
// steps square it to below double rounding, 2^-52 in all.  The range is tested once a
// panel by the caller: a division for the others here made 20 OC iterations of a 60x20
// grid 9% longer (18.8 -> 20.6 ms), a test of every pivot 1.4%.
__device__ __forceinline__ double td_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = r * (2.0 - x * r);
  return r * (2.0 - x * r);
}

}  // namespace tptfem
