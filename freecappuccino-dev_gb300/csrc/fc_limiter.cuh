// Slope limiters of the cell gradients (gradients.f90:141-160, applied by
// grad_scalar_field after every gradient when `limiter` is set), written
// once per cell for the CUDA kernels (fc_limiter.cu, built without FMA
// contraction) and for the host replay that checks them against the oracle
// (tests/replay/limiter_replay.cpp, built -ffp-contract=off).  Arrays are
// 0-based; the gradient is SoA: g[c], g[nT + c], g[2 nT + c].
//
//  FC_LIMITER_BJ     Barth-Jespersen        gradients.f90:288-366
//  FC_LIMITER_VENKAT Venkatakrishnan        gradients.f90:373-451
//  FC_LIMITER_R      the 'R3' case, whose active line is the R4 function
//                                           gradients.f90:456-535
//  FC_LIMITER_MD     multidimensional       gradients.f90:541-656
//
// The first three scale a cell's gradient by the smallest limiter value over
// its CSR row (the neighbours), with r = (global max or min of phi over the
// cells - phi_c) / (g_c . (x_n - x_c)) and r = 1 where |g_c . d| < 1.e-6 (a
// default-real literal, compared in double).  The multidimensional limiter
// corrects the gradient face by face, in ascending inner-face order, so one
// thread per cell walking its faces in that order reproduces the reference's
// face loop exactly.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define FC_HD __host__ __device__ __forceinline__
#else
#define FC_HD inline
#endif

// the values of fc_gpu.h
#ifndef FC_LIMITER_NONE
#define FC_LIMITER_NONE 0
#define FC_LIMITER_BJ 1
#define FC_LIMITER_VENKAT 2
#define FC_LIMITER_R 3
#define FC_LIMITER_MD 4
#endif

namespace fclim {

// the literal 1.e-6 of the reference's comparison: a single-precision
// constant, promoted to double
constexpr double kTinyDelta = (double)1.e-6f;

FC_HD double dmin(double a, double b) { return b < a ? b : a; }
FC_HD double dmax(double a, double b) { return b > a ? b : a; }

// limiter function of r for the three scaling limiters
template <int KIND>
FC_HD double limiter_fn(double r) {
  if (KIND == FC_LIMITER_BJ) return r;
  if (KIND == FC_LIMITER_VENKAT) return (r * r + 2.0 * r) / (r * r + r + 2.0);
  const double r2 = r * r, r3 = r2 * r, r4 = r2 * r2;
  return (r4 + 2.0 * r3 - 4.0 * r2 + 8.0 * r) / (r4 + r3 + 2.0 * r2 - 4.0 * r + 8.0);
}

// r from which limiter_fn is 1 or more, so that the neighbour does not lower the
// scale factor: 1 for BJ; 2 for VENKAT (numerator - denominator = r - 2) and
// for R ((r - 2)^3).  One per cent on top is far more than limiter_fn's and
// the screening's rounding.
template <int KIND>
constexpr float kFreeRatio = KIND == FC_LIMITER_BJ ? 1.01f : 2.02f;

// scale factor of cell c's gradient (gx, gy, gz) for KIND in BJ, VENKAT, R;
// fimin/fimax: min/max of phi over all cells
//
// A neighbour is screened first: the projection d in FP32 with a bound of its
// error (the coordinates' rounding and six more).  If it is certain that |d| is
// above kTinyDelta and r above kFreeRatio, the limiter value is 1 or more and
// the neighbour is passed over; if |d| is certainly below kTinyDelta, r is 1.
// NaN and infinities fail both tests.  The others are evaluated in FP64 as
// written: 38 FP64 instructions, two divisions among them, at 17 cycles a warp,
// which bounded the kernel; the screening takes three conversions.  fc_grad at
// 128^3, least squares with Venkatakrishnan, a smooth front with noise: 1,483 us
// without it (the limiter 1,005), 650 with the differences in FP64, now 607.
template <int KIND>
FC_HD double limit_factor(int c, const int* ia, const int* ja, const int* dg, const double* xc, const double* yc,
                          const double* zc, const double* phi, double gx, double gy, double gz, double fimin,
                          double fimax) {
  const double deltamax = fimax - phi[c];
  const double deltamin = fimin - phi[c];
  const double x = xc[c], y = yc[c], z = zc[c];
  const float gxf = (float)gx, gyf = (float)gy, gzf = (float)gz, room_up = (float)deltamax, room_dn = -(float)deltamin;
  const float xf = (float)x, yf = (float)y, zf = (float)z;
  const float ex = 1.e-7f * fabsf(gxf), ey = 1.e-7f * fabsf(gyf), ez = 1.e-7f * fabsf(gzf);
  double slopelimit = 1.0;
  const int kd = dg[c];
  for (int k = ia[c]; k < ia[c + 1]; ++k) {
    if (k == kd) continue;
    const int n = ja[k];
    const double xn = xc[n], yn = yc[n], zn = zc[n];
    const float xnf = (float)xn, ynf = (float)yn, znf = (float)zn;
    const float px = gxf * (xnf - xf), py = gyf * (ynf - yf), pz = gzf * (znf - zf);
    const float d = px + py + pz, size = fabsf(d);
    const float err = 1.e-6f * (fabsf(px) + fabsf(py) + fabsf(pz)) + ex * (fabsf(xnf) + fabsf(xf)) +
                      ey * (fabsf(ynf) + fabsf(yf)) + ez * (fabsf(znf) + fabsf(zf)) + 1.e-30f;
    if (size + err < 0.9e-6f) {
      slopelimit = dmin(slopelimit, limiter_fn<KIND>(1.0));
      continue;
    }
    if (size - err > 1.1e-6f && kFreeRatio<KIND> * (size + err) < (d > 0.f ? room_up : room_dn)) continue;
    const double delta_face = gx * (xn - x) + gy * (yn - y) + gz * (zn - z);
    if ((delta_face < 0.0 ? -delta_face : delta_face) < kTinyDelta) {
      slopelimit = dmin(slopelimit, limiter_fn<KIND>(1.0));
      continue;
    }
    slopelimit = dmin(slopelimit, limiter_fn<KIND>((delta_face > 0.0 ? deltamax : deltamin) / delta_face));
  }
  return slopelimit;
}

// multidimensional limiter of cell c: its gradient corrected face by face
// over its inner faces in ascending order (cf_face ascending, boundary faces
// f >= nI skipped); phimax/phimin over the cell's CSR row in row order
FC_HD void limit_md(int c, const int* ia, const int* ja, const int* cf_ptr, const int* cf_face, int nI,
                    const double* xf, const double* yf, const double* zf, const double* xc, const double* yc,
                    const double* zc, const double* phi, double& gx, double& gy, double& gz) {
  double phimax = phi[ja[ia[c]]], phimin = phimax;
  for (int k = ia[c] + 1; k < ia[c + 1]; ++k) {
    phimax = dmax(phimax, phi[ja[k]]);
    phimin = dmin(phimin, phi[ja[k]]);
  }
  const double pc = phi[c];
  const double dPhimax = phimax - pc, dPhimin = phimin - pc;
  for (int q = cf_ptr[c]; q < cf_ptr[c + 1]; ++q) {
    const int f = cf_face[q];
    if (f >= nI) continue;
    const double xpn = xf[f] - xc[c], ypn = yf[f] - yc[c], zpn = zf[f] - zc[c];
    const double dpn = sqrt(xpn * xpn + ypn * ypn + zpn * zpn);
    const double nx = xpn / dpn, ny = ypn / dpn, nz = zpn / dpn;
    const double gn = gx * nx + gy * ny + gz * nz;
    const double gtx = gx - gn * nx, gty = gy - gn * ny, gtz = gz - gn * nz;
    const double dPhi = gx * xpn + gy * ypn + gz * zpn;
    if (phimax > pc && dPhi > dPhimax) {
      gx = gtx + nx * dPhimax;
      gy = gty + ny * dPhimax;
      gz = gtz + nz * dPhimax;
    }
    if (phimin < pc && dPhi < dPhimin) {
      gx = gtx + nx * dPhimin;
      gy = gty + ny * dPhimin;
      gz = gtz + nz * dPhimin;
    }
  }
}

}  // namespace fclim
