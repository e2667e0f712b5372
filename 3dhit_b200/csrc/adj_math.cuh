// Per-mode arithmetic of the discrete adjoint (k_adjoint.cu, k_xadj.cu).
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace hit {

template <typename T> struct Mode {
  T kx, ky, kz, k2, ik2;
  int w;       // Hermitian weight
  bool keep;   // inside the 2/3 box (dealias mask)
};

template <typename T>
__device__ __forceinline__ Mode<T> mode_of(long long m, const Geom& g, const KTab<T>& kt, int& fx, int& fy, int& z) {
  z = (int)(m % g.Nzh);
  const long long r = m / g.Nzh;
  fy = (int)(r % g.Ny);
  fx = (int)(r / g.Ny);
  Mode<T> d;
  d.kx = kt.kx[fx];
  d.ky = kt.ky[fy];
  d.kz = kt.kz[z];
  d.k2 = k2_of(d.kx, d.ky, d.kz);
  d.ik2 = inv_k2_of(d.k2);
  d.w = herm_weight(g, z);
  d.keep = in_dealias(g, fx, fy, z);
  return d;
}

// project(dealias(v)) of one mode, in the reference's operation order
// (src/hit3d/grid.py:166-178)
template <typename T> __device__ __forceinline__ void proj_mask(const Mode<T>& d, V2<T> (&v)[3]) {
  if (!d.keep) {
    v[0] = v[1] = v[2] = czero<T>();
    return;
  }
  V2<T> div;
  div.x = (d.kx * v[0].x + d.ky * v[1].x + d.kz * v[2].x) * d.ik2;
  div.y = (d.kx * v[0].y + d.ky * v[1].y + d.kz * v[2].y) * d.ik2;
  v[0] = csub(v[0], cscale(div, d.kx));
  v[1] = csub(v[1], cscale(div, d.ky));
  v[2] = csub(v[2], cscale(div, d.kz));
}

template <typename T> __device__ __forceinline__ double re_dot3(const V2<T> (&a)[3], const V2<T> (&b)[3]) {
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) s += (double)a[c].x * b[c].x + (double)a[c].y * b[c].y;
  return s;
}

// 1j k x a
template <typename T> __device__ __forceinline__ void curl_of(const Mode<T>& d, const V2<T> (&a)[3], V2<T> (&o)[3]) {
  V2<T> t[3];
  t[0].x = d.ky * a[2].x - d.kz * a[1].x;
  t[0].y = d.ky * a[2].y - d.kz * a[1].y;
  t[1].x = d.kz * a[0].x - d.kx * a[2].x;
  t[1].y = d.kz * a[0].y - d.kx * a[2].y;
  t[2].x = d.kx * a[1].x - d.ky * a[0].x;
  t[2].y = d.kx * a[1].y - d.ky * a[0].y;
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = cmul_i(t[c]);
}

// Scalars of the forcing transpose from the six sums (one thread):
//   scal[0] a_all  (pv coefficient, every mode)   scal[1] a_band (pv coefficient, band)
//   scal[2] c_w    (coefficient of w u)           scal[3] c_wk2  (of w k2 u)
//   scal[4] c_wb   (of w u over the band)
// and the parameter cotangents pct[0] nu, pct[1] A, pct[2] eps (added).
__device__ __forceinline__ void adj_coef(const AdjCoefArgs& a, const double* s) {
  const double n2 = a.ntot2;
  double sc[5] = {0, 0, 0, 0, 0};
  double dnu = -s[2], dA = 0.0, deps = 0.0;
  if (a.forcing == 1) {  // f = A u (forcing.py:94-95)
    sc[0] = a.A;
    dA = s[0];
  } else if (a.forcing == 2) {  // f = c mask u, c = eps / 2E_band (forcing.py:138-143)
    const double twoE = s[5] / n2;
    if (twoE > a.tiny) {
      const double c = a.eps / twoE;
      sc[1] = c;
      sc[4] = s[1] * (-c / twoE) * 2.0 / n2;
      deps = s[1] / twoE;
    }
  } else if (a.forcing == 3) {  // f = A(u) u, A = (2 nu Omega - (E - E_t)/tau) / 2E
    const double E = s[3] / (2.0 * n2), Om = s[4] / (2.0 * n2);
    if (E > 0.0) {
      const double itau = (a.tau > 0.0 && isfinite(a.tau)) ? 1.0 / a.tau : 0.0;
      const double relax = (a.tau > 0.0 && isfinite(a.tau)) ? (E - a.E_target) / a.tau : 0.0;
      const double A = (2.0 * a.nu * Om - relax) / (2.0 * E);
      const double beta = s[0];
      sc[0] = A;
      sc[2] = beta / n2 * (-itau / (2.0 * E) - A / E);
      sc[3] = beta / n2 * (a.nu / E);
      dnu += beta * Om / E;
    }
  }
  for (int i = 0; i < 5; ++i) a.scal[i] = sc[i];
  a.pct[0] += dnu;
  a.pct[1] += dA;
  a.pct[2] += deps;
}

}  // namespace hit
