// k_plane: the middle of the RHS (y-inverse, z pass, y-forward; the work of
// k_axis, k_zwarp / k_zcross and k_axis) for planes that fit in shared memory:
// one CTA per x position takes the (y, z) plane of u and w through all of it
// and writes the three products' plane back in place.
//
// What bounds small grids is the chain of dependent launches: at 32^3 each of
// the three kernels took 4-5 us of mostly start-up, drain and L2 round trips.
// Here the plane crosses shared memory in seven phases with a barrier between
// them (RK4 step inside a rollout: 32^3 float32 67 -> 53 us, 64^3 107 -> 93, 64^3
// float64 160 -> 121; 512 x 32 x 32 334 -> 208; no shape served is slower; plain
// prefetches in the x passes later took the 32^3 step to 37).
// The transforms are two-stage (N = R0 x R1) and in place: the inverse
// ones decimate in frequency and leave their output permuted (index k at slot
// (k mod R0) R1 + k / R0), u x w is formed value by value in that order, and
// the forward ones decimate in time from it back to natural order, so no stage
// needs a second buffer or a second barrier:
//   1  y-inverse, stage over stride R1 (rows from global memory, zero-padded)
//   2  y-inverse, stage inside the blocks of R1
//   3  z c2r pre-processing and stage over stride R1 (bins k and H - k are
//      read by one thread, which owns both butterflies)
//   4  z block stage of u and w, u x w, z block stage of the products
//   5  z-forward, stage over stride R1
//   6  r2c post-processing (columns k and H - k by one thread) and y-forward
//      block stage
//   7  y-forward, stage over stride R1, to global memory
// Dealiased layout only (compile-time bounds).  STAGE: the plane's six fields
// (one contiguous run each) come in by bulk TMA copies first; used when a CTA
// has an SM to itself anyway, the staging rows being a third of its memory.
#include <type_traits>

#include "tma.cuh"
#include "xfield.cuh"

namespace hit {

constexpr int PLANE_WAIT = 1 << 22;  // mbarrier polls before a TMA wait gives up
__device__ int g_plane_timeout = 0;  // set when a TMA wait gave up (hit_device_status)
__device__ int g_plane_wait_limit = PLANE_WAIT;  // polls of the wait for a plane (hit_set_wait_limit)

cudaError_t set_plane_wait_limit(int polls) {
  const int v = polls < 0 ? PLANE_WAIT : polls;
  return cudaMemcpyToSymbol(g_plane_wait_limit, &v, sizeof(int));
}
cudaError_t take_plane_timeout(int* flag) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_plane_timeout, sizeof(int));
  if (e != cudaSuccess) return e;
  *flag = v;
  const int zero = 0;
  return v ? cudaMemcpyToSymbol(g_plane_timeout, &zero, sizeof(int)) : cudaSuccess;
}

template <int NY, int H> struct PlaneCfg {
  static constexpr int ZP = H + 1;                  // row pitch: odd, so lanes along y hit all banks
  static constexpr int MZ = (2 * H) / 3 + 1;        // stored z modes
  static constexpr int MZP = (MZ + 7) / 8 * 8;
  static constexpr int MY = 2 * (NY / 3) + 1;
  static constexpr int TW = NY + H + H + 1;         // w_NY^m, w_H^m, e^{-2 pi i k / 2H}
  static constexpr int SLOTS = (6 * NY * ZP + TW + 1) / 2 * 2;
  static constexpr int STG = 6 * MY * MZP;          // staged rows
};
template <typename T> __host__ __device__ constexpr int plane_threads() { return sizeof(T) == 4 ? 384 : 256; }

template <typename T, int NY, int H, bool STAGE>
__global__ void __launch_bounds__(plane_threads<T>()) k_plane(PlaneArgs<T> a) {
  using C = PlaneCfg<NY, H>;
  constexpr int NTH = plane_threads<T>();
  constexpr int Y0 = Two<NY>::R0, Y1 = Two<NY>::R1, Z0 = Two<H>::R0, Z1 = Two<H>::R1;
  constexpr int ZP = C::ZP, MZ = C::MZ, MZP = C::MZP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<T>* P = reinterpret_cast<V2<T>*>(smem_raw);  // [field][y slot][z slot]
  V2<T>* twy = P + 6 * NY * ZP;
  V2<T>* twh = twy + NY;
  V2<T>* twz = twh + H;
  for (int e = threadIdx.x; e < C::TW; e += NTH)
    twy[e] = e < NY ? a.tw[e * (TWN / NY)] : (e < NY + H ? a.tw[(e - NY) * (TWN / H)] : a.tw[(e - NY - H) * (TWN / (2 * H))]);
  auto at = [&](int f, int y, int z) -> V2<T>& { return P[(f * NY + y) * ZP + z]; };
  auto cw = [](V2<T> v, V2<T> w) {  // v conj(w)
    w.y = -w.y;
    return cmul(v, w);
  };
  V2<T>* plane = a.t6 + (long long)blockIdx.x * a.t_x;
  V2<T>* stg = P + C::SLOTS;
  __shared__ __align__(8) uint64_t bar;
  const uint32_t mb = tma::smem_u32(&bar);
  const int wait_limit = STAGE ? g_plane_wait_limit : 0;
  if (STAGE && threadIdx.x == 0) tma::mbar_init(mb, 1);
  pdl_wait();
  pdl_trigger();
  if constexpr (STAGE) {
    constexpr uint32_t FB = C::MY * MZP * (uint32_t)sizeof(V2<T>);
    if (threadIdx.x == 0) {
      tma::mbar_expect_tx(mb, 6 * FB);
      for (int f = 0; f < 6; ++f) tma::load_bytes(stg + f * C::MY * MZP, plane + f * a.t_c, FB, mb);
    }
    __syncthreads();  // the barrier's initialisation and the twiddles
    if (!__syncthreads_and(tma::mbar_wait(mb, 0, wait_limit))) {
      if (threadIdx.x == 0) atomicExch(&g_plane_timeout, 1);
      tma::mbar_wait(mb, 0, PLANE_WAIT);  // the copies in flight, once more with a limit
      return;
    }
  } else {
    __syncthreads();  // the twiddles
  }
  // 1
  {
    Geom unused{};
    const XRows<NY, true> rows(unused);
    for (int t = threadIdx.x; t < 6 * Y1 * MZ; t += NTH) {
      const int z = t % MZ, b = t / MZ % Y1, f = t / MZ / Y1;
      const V2<T>* src = (STAGE ? stg + f * C::MY * MZP : plane + f * a.t_c) + z;
      V2<T> v[Y0];
#pragma unroll
      for (int r = 0; r < Y0; ++r) {
        const int row = rows.row(b, r * Y1, Y1);
        v[r] = row >= 0 ? src[row * MZP] : czero<T>();
      }
      DFT<Y0, true, V2<T>>::run(v);
#pragma unroll
      for (int k = 0; k < Y0; ++k) at(f, k * Y1 + b, z) = k ? cw(v[k], twy[b * k]) : v[k];
    }
  }
  __syncthreads();
  // 2
  for (int t = threadIdx.x; t < 6 * Y0 * MZ; t += NTH) {
    const int z = t % MZ, k0 = t / MZ % Y0, f = t / MZ / Y0;
    V2<T> v[Y1];
#pragma unroll
    for (int b = 0; b < Y1; ++b) v[b] = at(f, k0 * Y1 + b, z);
    DFT<Y1, true, V2<T>>::run(v);
#pragma unroll
    for (int b = 0; b < Y1; ++b) at(f, k0 * Y1 + b, z) = v[b];
  }
  __syncthreads();
  // 3
  for (int t = threadIdx.x; t < 6 * (Z1 / 2 + 1) * NY; t += NTH) {
    const int y = t % NY, b = t / NY % (Z1 / 2 + 1), f = t / NY / (Z1 / 2 + 1);
    const int bb = b == 0 ? 0 : Z1 - b;
    V2<T>* row = P + (f * NY + y) * ZP;
    // e^{+2 pi i k / Nz} pre-processing of bin k from X = X[k] and Y = X[H - k]
    auto pre = [&](int k, V2<T> X, V2<T> Y) {
      if (k == 0) {
        X.y = T(0);
        Y.y = T(0);
      }
      Y.y = -Y.y;
      return cadd(cadd(X, Y), cmul_i(cw(csub(X, Y), twz[k])));
    };
    auto ld = [&](int k) { return k < MZ ? row[k] : czero<T>(); };
    V2<T> xa[Z0], xb[Z0], za[Z0], zb[Z0];
#pragma unroll
    for (int r = 0; r < Z0; ++r) {
      xa[r] = ld(b + r * Z1);
      xb[r] = ld(bb + r * Z1);
    }
    const V2<T> xh = b == 0 ? ld(H) : czero<T>();
#pragma unroll
    for (int r = 0; r < Z0; ++r) {
      za[r] = pre(b + r * Z1, xa[r], b == 0 ? (r == 0 ? xh : xa[(Z0 - r) % Z0]) : xb[Z0 - 1 - r]);
      zb[r] = pre(bb + r * Z1, xb[r], xa[Z0 - 1 - r]);  // used when bb is another butterfly
    }
    DFT<Z0, true, V2<T>>::run(za);
#pragma unroll
    for (int k = 0; k < Z0; ++k) row[k * Z1 + b] = k ? cw(za[k], twh[b * k]) : za[k];
    if (bb != b) {
      DFT<Z0, true, V2<T>>::run(zb);
#pragma unroll
      for (int k = 0; k < Z0; ++k) row[k * Z1 + bb] = k ? cw(zb[k], twh[bb * k]) : zb[k];
    }
  }
  __syncthreads();
  // 4
  const T s2 = T(0.5) * a.scale * a.scale;  // both inverse normalisations and the r2c 1/2
  for (int t = threadIdx.x; t < NY * Z0; t += NTH) {
    const int y = t % NY, k0 = t / NY;
    V2<T> v[6][Z1];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
#pragma unroll
      for (int b = 0; b < Z1; ++b) v[f][b] = at(f, y, k0 * Z1 + b);
      DFT<Z1, true, V2<T>>::run(v[f]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {  // u x w (navierstokes.py:82-86)
      const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
      V2<T> n[Z1];
#pragma unroll
      for (int b = 0; b < Z1; ++b) {
        n[b].x = (v[c1][b].x * v[3 + c2][b].x - v[c2][b].x * v[3 + c1][b].x) * s2;
        n[b].y = (v[c1][b].y * v[3 + c2][b].y - v[c2][b].y * v[3 + c1][b].y) * s2;
      }
      DFT<Z1, false, V2<T>>::run(n);
#pragma unroll
      for (int b = 0; b < Z1; ++b) at(c, y, k0 * Z1 + b) = b ? cmul(n[b], twh[k0 * b]) : n[b];
    }
  }
  __syncthreads();
  // 5
  for (int t = threadIdx.x; t < 3 * Z1 * NY; t += NTH) {
    const int y = t % NY, b = t / NY % Z1, c = t / NY / Z1;
    V2<T> v[Z0];
#pragma unroll
    for (int k = 0; k < Z0; ++k) v[k] = at(c, y, k * Z1 + b);
    DFT<Z0, false, V2<T>>::run(v);
#pragma unroll
    for (int k = 0; k < Z0; ++k) at(c, y, k * Z1 + b) = v[k];
  }
  __syncthreads();
  // 6
  for (int t = threadIdx.x; t < 3 * Y0 * (H / 2 + 1); t += NTH) {
    const int p = t % (H / 2 + 1), k0 = t / (H / 2 + 1) % Y0, c = t / (H / 2 + 1) / Y0;
    const int q = H - p;
    const bool two = q < MZ && q != p;  // the partner column is stored too
    const V2<T> wp = twz[p], wq = twz[q];
    V2<T> x[Y1], xq[Y1];
#pragma unroll
    for (int b = 0; b < Y1; ++b) {
      const V2<T> za = at(c, k0 * Y1 + b, p), zb = at(c, k0 * Y1 + b, p == 0 ? 0 : q);
      const V2<T> ca = cconj(za), cb = cconj(zb);
      x[b] = cadd(cadd(za, cb), cmul(wp, cmul_mi(csub(za, cb))));
      xq[b] = cadd(cadd(zb, ca), cmul(wq, cmul_mi(csub(zb, ca))));
    }
    DFT<Y1, false, V2<T>>::run(x);
#pragma unroll
    for (int b = 0; b < Y1; ++b) at(c, k0 * Y1 + b, p) = b ? cmul(x[b], twy[k0 * b]) : x[b];
    if (two) {
      DFT<Y1, false, V2<T>>::run(xq);
#pragma unroll
      for (int b = 0; b < Y1; ++b) at(c, k0 * Y1 + b, q) = b ? cmul(xq[b], twy[k0 * b]) : xq[b];
    }
  }
  __syncthreads();
  // 7
  {
    Geom unused{};
    const XRows<NY, true> rows(unused);
    for (int t = threadIdx.x; t < 3 * Y1 * MZP; t += NTH) {
      const int z = t % MZP, b = t / MZP % Y1, c = t / MZP / Y1;
      V2<T> v[Y0];
#pragma unroll
      for (int k = 0; k < Y0; ++k) v[k] = z < MZ ? at(c, k * Y1 + b, z) : czero<T>();
      DFT<Y0, false, V2<T>>::run(v);
      V2<T>* dst = plane + c * a.t_c + z;
#pragma unroll
      for (int k = 0; k < Y0; ++k) {
        const int row = rows.row(b, k * Y1, Y1);
        if (row >= 0) dst[row * MZP] = v[k];
      }
    }
  }
}

template <typename T, int NY, int H, bool STAGE> cudaError_t launch_plane_v(const PlaneArgs<T>& a, cudaStream_t st) {
  using C = PlaneCfg<NY, H>;
  constexpr size_t smem = sizeof(V2<T>) * (size_t)(C::SLOTS + (STAGE ? C::STG : 0));
  if constexpr (STAGE && smem > 220 * 1024) {
    return launch_plane_v<T, NY, H, false>(a, st);
  } else {
    static_assert(smem <= 220 * 1024, "plane_fits");
    static PerDevice ready;
    cudaError_t e = once_per_device(ready, [] { return xf_attr(k_plane<T, NY, H, STAGE>, smem); });
    if (e != cudaSuccess) return e;
    return launch_pdl(k_plane<T, NY, H, STAGE>, a.g.Nx, plane_threads<T>(), smem, st, a);
  }
}
template <typename T, int NY, int H> cudaError_t launch_plane_s(const PlaneArgs<T>& a, cudaStream_t st) {
  return a.g.Nx <= 148 ? launch_plane_v<T, NY, H, true>(a, st) : launch_plane_v<T, NY, H, false>(a, st);
}

template <typename T> cudaError_t launch_plane(const PlaneArgs<T>& a, cudaStream_t st) {
  auto by_ny = [&](auto hh) {
    constexpr int H = decltype(hh)::value;
    switch (a.g.Ny) {
      case 8: return launch_plane_s<T, 8, H>(a, st);
      case 16: return launch_plane_s<T, 16, H>(a, st);
      case 32: return launch_plane_s<T, 32, H>(a, st);
      case 64: return launch_plane_s<T, 64, H>(a, st);
      default: return cudaErrorInvalidValue;
    }
  };
  switch (a.g.H) {
    case 4: return by_ny(std::integral_constant<int, 4>{});
    case 8: return by_ny(std::integral_constant<int, 8>{});
    case 16: return by_ny(std::integral_constant<int, 16>{});
    case 32: return by_ny(std::integral_constant<int, 32>{});
    default: return cudaErrorInvalidValue;
  }
}

bool plane_fits(const Geom& g) {
  return g.pruned && g.Ny >= 8 && g.Ny <= 64 && g.Nz >= 8 && g.Nz <= 64;
}

template cudaError_t launch_plane<float>(const PlaneArgs<float>&, cudaStream_t);
template cudaError_t launch_plane<double>(const PlaneArgs<double>&, cudaStream_t);

}  // namespace hit
