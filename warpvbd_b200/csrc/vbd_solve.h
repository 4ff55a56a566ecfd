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

// 1 / x for 2^-1000 < x < 2^1000: on the device the hardware's approximation and
// newton_reciprocal.
VBD_HOST_DEVICE double reciprocal64(double x) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return newton_reciprocal(x, y);
#else
  return 1.0 / x;
#endif
}

VBD_HOST_DEVICE double dot3(double a0, double b0, double a1, double b1, double a2, double b2) {
  return fma(a2, b2, fma(a1, b1, a0 * b0));
}
VBD_HOST_DEVICE double cross2(double a, double b, double c, double d) {  // ab - cd
  return fma(a, b, -(c * d));
}

// Solves H x = -g (h = h00 h01 h02 h11 h12 h22) by H = L D L^T; false when a pivot is not
// positive (H not positive definite).
VBD_HOST_DEVICE bool ldl_solve3(const double* h, const double* g, double* x) {
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

// The same: one step of the elimination, the 2x2 block left (times h00) by Cramer's rule,
// which is forward stable at that size.  The error grows with the condition number, as that of
// the Cholesky form the reference takes (tile_cholesky, vbd_solver.py:267-268), not with its
// square as the 3x3 cofactor form's: a nearly incompressible tet has one direction lambda / mu
// times stiffer than the others.  Median relative error of H = random + k c c^T at
// k = 1 / 1e3 / 1e5 / 1e9: 1.0e-16 / 4.3e-15 / 4.3e-13 / 4.4e-9 here, 1.0e-16 / 3.9e-15 /
// 3.9e-13 / 4.0e-9 by L D L^T, 1.7e-16 / 6.5e-15 / 5.7e-13 / 5.7e-9 by Cholesky, 1.3e-16 /
// 8.6e-14 / 7.9e-10 / 8.1e-2 by 3x3 cofactors.  One lane per vertex runs it while the warp
// waits: its chain has one reciprocal, L D L^T's three (us per sweep here / by L D L^T / by 3x3
// cofactors: 20x2x2 beam 13.5 / 14.1 / 13.2, 80x8x8 StVK beam 18.0 / 18.7 / 17.7, 160x16x16
// beam 31.0 / 31.8 / 31.7).  What is not clearly positive definite, or leaves the range of the
// products, goes by L D L^T.
VBD_HOST_DEVICE bool solve3(const double* h, const double* g, double* x) {
  const double p1 = cross2(h[0], h[3], h[1], h[1]), p2 = cross2(h[0], h[5], h[2], h[2]),
               q = cross2(h[0], h[4], h[1], h[2]);
  const double det = cross2(p1, p2, q, q);  // h00 times H's
  if (!(h[0] > 1e-250 && h[0] < 1e250 && p1 > 0.0 && det > 1e-250 && det < 1e250))
    return ldl_solve3(h, g, x);
  const double r = reciprocal64(det), i0 = reciprocal64(h[0]);
  const double y1 = cross2(h[1], g[0], h[0], g[1]), y2 = cross2(h[2], g[0], h[0], g[2]);
  x[1] = mul_rounded(cross2(p2, y1, q, y2), r);
  x[2] = mul_rounded(cross2(p1, y2, q, y1), r);
  x[0] = mul_rounded(fma(-h[2], x[2], fma(-h[1], x[1], -g[0])), i0);
  return true;
}

}  // namespace vbd
