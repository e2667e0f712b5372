// RHS epilogue of one spectral mode, shared by the x-forward kernels
// (k_axis.cu, k_xfield.cu): state loads, then forcing, dealias mask,
// projection, viscous term, RK4 stage algebra and the float64 partial sums.
#pragma once

#include "common.cuh"
#include "kernels.h"

namespace hit {

// Element o of a component's array: a 32-bit byte offset from a base that is
// uniform over the block (one address register instead of 64-bit arithmetic
// per access; callers use it when a component is smaller than 4 GB) or a
// 64-bit element offset.
template <typename V> __device__ __forceinline__ V& elem(V* base, uint32_t byte_off) {
  return *reinterpret_cast<V*>(reinterpret_cast<char*>(base) + byte_off);
}
template <typename V> __device__ __forceinline__ const V& elem(const V* base, uint32_t byte_off) {
  return *reinterpret_cast<const V*>(reinterpret_cast<const char*>(base) + byte_off);
}
template <typename V> __device__ __forceinline__ V& elem(V* base, long long o) { return base[o]; }
template <typename V> __device__ __forceinline__ const V& elem(const V* base, long long o) { return base[o]; }

// State rows of one mode for the epilogue: us = stage input (u for stages
// 0/1), ac/uu = accumulator and u (stages 2..4).
template <typename T, typename OFF>
__device__ __forceinline__ void p3_load(const P3Args<T>& a, OFF o, V2<T> (&us)[3], V2<T> (&ac)[3],
                                        V2<T> (&uu)[3]) {
  const V2<T>* __restrict__ pus = a.stage <= 1 ? a.u : a.s;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    us[c] = elem(pus + c * a.c_c, o);
    if (a.stage >= 2) {
      ac[c] = elem(a.acc + c * a.c_c, o);
      uu[c] = elem(a.u + c * a.c_c, o);
    }
  }
}

// RHS epilogue of one stored mode (x position pos, z index z, state offset
// o): du holds the x-forward nonlinear term (u x w)^ on entry.  Forcing is
// added before dealias and projection (navierstokes.py:88-92), then the
// viscous term (navierstokes.py:95) and the RK4 stage algebra
// (integrators.py:32-38); ns receives the new stage input (or new state) and
// the float64 partial sums are accumulated.
template <typename T, typename OFF>
__device__ __forceinline__ void p3_point(const P3Args<T>& a, int pos, int fy, int z, T ky, T kz, T cf, OFF o,
                                         V2<T> (&du)[3], const V2<T> (&us)[3], const V2<T> (&ac)[3],
                                         const V2<T> (&uu)[3], V2<T> (&ns)[3], double& sE, double& sO,
                                         double& sB) {
  const Geom& g = a.g;
  const T kx = __ldg(a.k.kx + pos);
  const T k2 = k2_of(kx, ky, kz);
  const T ik2 = inv_k2_of(k2);
  if (a.fext) {
#pragma unroll
    for (int c = 0; c < 3; ++c) du[c] = cadd(du[c], elem(a.fext + c * a.c_c, o));
  }
  if (a.forcing == 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) du[c] = cadd(du[c], cscale(us[c], a.fA));
  } else if (a.forcing == 2) {
    if (a.kmin2 <= k2 && k2 <= a.kmax2) {
#pragma unroll
      for (int c = 0; c < 3; ++c) du[c] = cadd(du[c], cscale(us[c], cf));
    }
  } else if (a.forcing == 3) {
#pragma unroll
    for (int c = 0; c < 3; ++c) du[c] = cadd(du[c], cscale(us[c], cf));
  }
  // every stored mode of the dealiased path lies inside the 2/3 box
  if (g.pruned ? (pos | fy | z) == 0 : !in_dealias(g, pos, fy, z)) {
    du[0] = du[1] = du[2] = czero<T>();
  }
  // projection: div = (kx d0 + ky d1 + kz d2) / k^2 ; d -= k div
  V2<T> div;
  div.x = (kx * du[0].x + ky * du[1].x + kz * du[2].x) * ik2;
  div.y = (kx * du[0].y + ky * du[1].y + kz * du[2].y) * ik2;
  du[0] = csub(du[0], cscale(div, kx));
  du[1] = csub(du[1], cscale(div, ky));
  du[2] = csub(du[2], cscale(div, kz));
  const T nk2 = a.nu * k2;
#pragma unroll
  for (int c = 0; c < 3; ++c) du[c] = csub(du[c], cscale(us[c], nk2));

  V2<T>* __restrict__ pu = a.u_out;
  V2<T>* __restrict__ pacc = a.acc;
  V2<T>* __restrict__ ps = a.s_out;
  V2<T>* __restrict__ pout = a.out;
  if (a.ifrk && a.stage > 0) {
    // integrating-factor (Lawson) RK4 with E = e^{-nu k^2 dt/2} and N the RHS
    // without its viscous term:
    //   s2 = E (u + dt/2 k1),  s3 = E u + dt/2 k2,  s4 = E^2 u + dt E k3,
    //   u' = E^2 u + dt/6 ((E (E k1 + 2 k2) + 2 E k3) + k4)
    // (acc holds E k1, then E (E k1 + 2 k2), then + 2 E k3)
    const T E = visc_factor(a.nuh, k2);
    switch (a.stage) {
      case 1:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          elem(pacc + c * a.c_c, o) = cscale(du[c], E);
          ns[c] = cscale(cadd(us[c], cscale(du[c], a.a_next)), E);
          elem(ps + c * a.c_c, o) = ns[c];
        }
        break;
      case 2:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          V2<T> acn = ac[c];
          acn.x = acn.x + T(2) * du[c].x;
          acn.y = acn.y + T(2) * du[c].y;
          elem(pacc + c * a.c_c, o) = cscale(acn, E);
          ns[c] = cadd(cscale(uu[c], E), cscale(du[c], a.a_next));
          elem(ps + c * a.c_c, o) = ns[c];
        }
        break;
      case 3:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const V2<T> ek = cscale(du[c], E);
          V2<T> acn = ac[c];
          acn.x = acn.x + T(2) * ek.x;
          acn.y = acn.y + T(2) * ek.y;
          elem(pacc + c * a.c_c, o) = acn;
          ns[c] = cadd(cscale(uu[c], E * E), cscale(ek, a.a_next));
          elem(ps + c * a.c_c, o) = ns[c];
        }
        break;
      default:
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const V2<T> acn = cadd(ac[c], du[c]);
          ns[c] = cadd(cscale(uu[c], E * E), cscale(acn, a.dt6));
          elem(pu + c * a.c_c, o) = ns[c];
        }
        break;
    }
  } else switch (a.stage) {
    case 0:
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        elem(pout + c * a.c_c, o) = du[c];
        ns[c] = czero<T>();
      }
      break;
    case 1:
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        elem(pacc + c * a.c_c, o) = du[c];
        ns[c] = cadd(us[c], cscale(du[c], a.a_next));
        elem(ps + c * a.c_c, o) = ns[c];
      }
      break;
    case 2:
    case 3:
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        V2<T> acn = ac[c];
        acn.x = acn.x + T(2) * du[c].x;
        acn.y = acn.y + T(2) * du[c].y;
        elem(pacc + c * a.c_c, o) = acn;
        ns[c] = cadd(uu[c], cscale(du[c], a.a_next));
        elem(ps + c * a.c_c, o) = ns[c];
      }
      break;
    default:
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const V2<T> acn = cadd(ac[c], du[c]);
        ns[c] = cadd(uu[c], cscale(acn, a.dt6));
        elem(pu + c * a.c_c, o) = ns[c];
      }
      break;
  }
  if (a.partial) {
    double a2 = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) a2 += (double)ns[c].x * ns[c].x + (double)ns[c].y * ns[c].y;
    const double w = herm_weight(g, z);
    sE += w * a2;
    sO += w * (double)k2 * a2;
    if (a.kmin2 <= k2 && k2 <= a.kmax2) sB += w * a2;
  }
}

}  // namespace hit
