// One point of DFI's polar-to-Cartesian regridding (shared by
// atb_dfi_regrid and the inverse transform that regrids its rows on the
// fly, so both compute the same values bit for bit).
//
// For Cartesian frequency (i, j) of the w x w grid: the unit-circle mask
// of make_circle_mask(w, 1.0) (algotom/util/utility.py, integer grid
// centred at w // 2), the polar coordinates of generate_mapping_coordinate
// (algotom/rec/reconstruction.py:687-728, height_rec = width_rec =
// width_sino = w: radius clipped to floor((w - 1) / 2), the half plane
// folded by the Hermitian symmetry of a real image's spectrum, angle
// scaled to the sinogram's rows, both rounded to float32 as the reference's
// maps are), then map_coordinates(order=5, mode="reflect") of the complex
// row spectra: 6 x 6 quintic B-spline taps of the coefficients with
// half-sample symmetric indices.  FP64.
#pragma once

#include <cmath>

namespace atb {
namespace dfi {

// The six weights of the centred quintic B-spline at distances t + 2, t + 1, t,
// 1 - t, 2 - t and 3 - t, 0 <= t < 1: its three polynomials, each where it
// holds, without branches or divisions (which took most of the FP64 work of a
// point).
__device__ __forceinline__ void bspline5_weights(double t, double (&w)[6]) {
  auto inner = [](double a) {  // a < 1
    const double a2 = a * a;
    return fma(a2, fma(a2, fma(a, -1.0 / 12.0, 0.25), -0.5), 0.55);
  };
  auto middle = [](double a) {  // 1 <= a < 2
    return fma(a, fma(a, fma(a, fma(a, fma(a, 1.0 / 24.0, -0.375), 1.25), -1.75), 0.625), 0.425);
  };
  auto outer = [](double b) {  // b = 3 - a
    const double b2 = b * b;
    return b2 * b2 * b * (1.0 / 120.0);
  };
  const double s = 1.0 - t;
  w[0] = outer(s);
  w[1] = middle(1.0 + t);
  w[2] = inner(t);
  w[3] = inner(s);
  w[4] = middle(1.0 + s);
  w[5] = outer(t);
}

// half-sample symmetric index
__device__ __forceinline__ int reflect_index(int i, int n) {
  if (i >= 0 && i < n) return i;
  const int p = 2 * n;
  int r = i % p;
  if (r < 0) r += p;
  return r >= n ? p - 1 - r : r;
}

// coef: complex B-spline coefficients [nrow][w], rows crs double2 apart
__device__ __forceinline__ double2 regrid_point(const double2 *__restrict__ coef, long long crs, int nrow, int w,
                                                int i, int j) {
  const long long cm = w / 2, dx = j - cm, dy = i - cm;
  if (dx * dx + dy * dy > cm * cm) return make_double2(0.0, 0.0);
  const double xc = (w - 1.0) * 0.5;
  const double rmax = floor(xc);
  const double x = (double)(w - 1 - j) - xc, y = (double)i - xc;
  float r = (float)fmin(fmax(sqrt(x * x + y * y), 0.0), rmax);
  double th = M_PI + atan2(y, x);
  if (th > M_PI) r = -r;
  r = (float)fmin(fmax((double)r + rmax, 0.0), (double)(w - 1));
  if (th > M_PI) th -= M_PI;
  const float tf = (float)(th * (nrow - 1.0) / M_PI);
  const double rr = (double)tf, cc = (double)r;
  const double rf = floor(rr), cf = floor(cc);
  const int fr = (int)rf - 2, fc = (int)cf - 2;
  double wr[6], wc[6];
  bspline5_weights(rr - rf, wr);
  bspline5_weights(cc - cf, wc);
  int ir[6], ic[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    ir[m] = reflect_index(fr + m, nrow);
    ic[m] = reflect_index(fc + m, w);
  }
  double re = 0.0, im = 0.0;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const double2 *row = coef + (long long)ir[a] * crs;
    double sr = 0.0, si = 0.0;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
      const double2 v = __ldg(row + ic[b]);
      sr += wc[b] * v.x;
      si += wc[b] * v.y;
    }
    re += wr[a] * sr;
    im += wr[a] * si;
  }
  return make_double2(re, im);
}

}  // namespace dfi
}  // namespace atb
