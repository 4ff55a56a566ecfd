// The fp64 3x3 solve of a vertex's Newton step, and the reciprocal of its slots.  Plain C++
// apart from one rounding intrinsic, so that it also compiles for the host.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define VBD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define VBD_HOST_DEVICE inline
#endif

namespace vbd {

// a b, rounded: never fused into an addition that follows.
VBD_HOST_DEVICE double mul_rounded(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

// 1 / x from an approximation y of 20 correct bits or more (rcp.approx.ftz.f64's): two Newton
// steps y (2 - x y), each of which squares the relative error.  The second adds less than
// 2^-79 / x to the rounding of the result.
VBD_HOST_DEVICE double newton_reciprocal(double x, double y) {
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// Solves H x = -g (h = h00 h01 h02 h11 h12 h22) by H = L D L^T; false when a pivot is not
// positive (H not positive definite).  Its error is that of the Cholesky form, which the
// reference takes (tile_cholesky, vbd_solver.py:267-268): backward stable, so it grows with
// the condition number, not with its square as the cofactor form's.  A nearly incompressible
// tet has one direction lambda / mu times stiffer than the others.  Median relative error of
// H = random + k c c^T at k = 1 / 1e3 / 1e5 / 1e9: 1.1e-16 / 3.9e-15 / 3.8e-13 / 3.9e-9
// here, 1.8e-16 / 6.3e-15 / 5.8e-13 / 5.6e-9 by Cholesky, 1.3e-16 / 8.6e-14 / 7.9e-10 / 8.1e-2
// by cofactors.  Without Cholesky's three square roots its chain, which one lane per vertex
// runs while the warp waits, is three reciprocals.
VBD_HOST_DEVICE bool solve3(const double* h, const double* g, double* x) {
  const double i0 = 1.0 / h[0];
  const double l10 = h[1] * i0, l20 = h[2] * i0;
  const double d1 = fma(-l10, h[1], h[3]), e = fma(-l20, h[1], h[4]);
  const double i1 = 1.0 / d1;
  const double l21 = e * i1;
  const double d2 = fma(-l21, e, fma(-l20, h[2], h[5]));
  const double i2 = 1.0 / d2;
  const double y1 = fma(l10, g[0], -g[1]);
  const double y2 = fma(-l21, y1, fma(l20, g[0], -g[2]));
  x[2] = mul_rounded(y2, i2);
  x[1] = fma(-l21, x[2], y1 * i1);
  x[0] = fma(-l20, x[2], fma(-l10, x[1], -(g[0] * i0)));
  return (h[0] > 0.0) && (d1 > 0.0) && (d2 > 0.0);
}

}  // namespace vbd
