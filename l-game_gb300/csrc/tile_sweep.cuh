// tile_sweep.cuh -- the two sequential sweeps of ks_column_ver_tile (split.cu) over a block's columns in
// shared memory, a lane per column: TC lanes, C the type of the coefficients.  A row holds kTileCoef
// coefficients, lane-interleaved: diagonal (then the pivot p), c, e (then e/p), and two the sweeps do not
// touch; a row of r holds the right-hand side.
#pragma once

#include "kernels.cuh"

namespace lg {

constexpr int kTileCoef = 5;

// wide() without its branches, for the sweep of a single warp: normal numbers; a zero becomes 2^-127, which
// beside the right-hand sides is none
__device__ __forceinline__ double wide_normal(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7FFFFFFFu;
  return __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (896u << 20))), (int)(a << 29));
}

// A pivot's reciprocal and the two quotients by it.  FP32: r to a unit of the last place (one instruction; the
// chain of pivots waits for it), e/p = e*r, and c/p as an FP64 number to 2^-45: c*r as the exact sum of two FP32
// numbers, the second with c times r's residual correction.  An FP32 multiplier c/p would be good to 2^-24 and
// carry that into right-hand sides that are held in FP64; it would save 1 % of a launch.  FP64: the rounded
// quotients.
__device__ __forceinline__ void quotients(float c, float e, float p, double* c_p, float* e_p) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p));
  const float r_lo = __fmaf_rn(-p, r, 1.f) * r, hi = c * r;
  *c_p = wide_normal(hi) + wide_normal(__fmaf_rn(c, r_lo, __fmaf_rn(c, r, -hi)));
  *e_p = e * r;
}
__device__ __forceinline__ void quotients(double c, double e, double p, double* c_p, double* e_p) {
  *c_p = c / p;
  *e_p = e / p;
}

// factorisation (pivot p, upper factor e/p, type C) and forward substitution of rows 1..n:
// y = r - (c/p)*y of the row above, one multiply-add a row in the chain
template <class C, int TC>
__device__ __forceinline__ void tile_forward(C* row, double* r, int n) {
  C cv_prev = C(0), epr_prev = C(0);
  double y = 0.0, f = 0.0;
#pragma unroll 4
  for (int jl = 1; jl <= n; ++jl, row += kTileCoef * TC, r += TC) {
    const C piv = row[0] - epr_prev * cv_prev;
    y = fma(-f, y, r[0]);
    r[0] = y;
    cv_prev = row[TC];
    quotients(cv_prev, row[2 * TC], piv, &f, &epr_prev);
    row[0] = piv;
    row[2 * TC] = epr_prev;
  }
}

// back substitution of rows n-1..1, r holding y/p; row, r: the first row's
template <class C, int TC>
__device__ __forceinline__ void tile_back(const C* row, double* r, int n) {
  row += kTileCoef * TC * (n - 2);
  r += TC * (n - 2);
  double s = r[TC];
#pragma unroll 4
  for (int jl = n - 1; jl >= 1; --jl, row -= kTileCoef * TC, r -= TC) {
    double e;
    if constexpr (sizeof(C) == 8) e = row[2 * TC];
    else e = wide(row[2 * TC]);
    s = fma(-e, s, r[0]);
    r[0] = s;
  }
}

}  // namespace lg
