// x-axis ends of the RHS for columns of at most 256 points (128 in float64),
// one thread group per transformed field: k_p3f (x-forward, RHS epilogue, RK4 stage update and
// the next stage's x-inverse; the work of k_p3) and k_p1f (x-inverse alone).
//
// A CTA owns a tile of all N x positions times W contiguous z columns of one
// ky row and has five groups of G threads.  Groups 0..2 run the three forward
// transforms of u x w side by side, all threads run the epilogue, and the five
// groups run the five inverse transforms (u_x, kx u_y, kx u_z, u_y, u_z) side
// by side; their outputs meet in shared memory, where w = i k x u is formed.
// Each transform is two stages (N = R0 x R1, at most 16 x 16), so it crosses
// shared memory once, and its one exchange is ordered by a barrier of the
// group alone.
//
// What bounded the column kernel before: at columns of 256 points and fewer
// k_p3 ran its eight transforms one after another with every thread of the
// CTA on each, three barriers per transform (about 35 per tile), half to three
// quarters of the threads without a butterfly in the radix-8 stages, and an
// instruction footprint that small grids fetched from L2 tile by tile (ncu:
// barrier and instruction-fetch stalls 8.9 + 4.6 per issue at 128 points, 12.5
// + 8.2 at 32).  Here a tile has about eight CTA barriers, the transforms'
// latencies overlap, and the layout's row bounds and 32-bit offsets fold most
// of the address arithmetic into constants (a quarter of the instructions).
// Time per launch of k_p3 -> k_p3f, stages with the fused x-inverse:
//   256^3 float32, hold-energy sums  309 -> 168 us (586 MB: 0.53 of HBM)
//   256^3 general layout             753 -> 547
//   128 x 64 x 256                    60 -> 27
//   64^3 hold-energy sums             31 -> 11
//   128^3 float64                    102 -> 56
// What bounds it now: the latency of a tile's two phases at two CTAs per SM.  A
// one-group form for columns of 256 points (16 values per thread, the spectral
// values in tensor memory, four CTAs per SM) measured 180 us and 20% more at
// few tiles.
#include "xfield.cuh"

namespace hit {

template <typename T, int N, int W, int G, int MINB, bool DA>
__global__ void __launch_bounds__(XF_GROUPS* G, MINB) k_p3f(P3Args<T> a, int nzt, int ntiles, int f_off) {
  using XT = XTile<N, W>;
  constexpr int NTH = XF_GROUPS * G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[96];
  V2<T>* tws = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* X = tws + XT::TWS;  // five exchange tiles
  V2<T>* F = X + f_off;      // 3 x Mx x W: the nonlinear term, then the new stage input
  const Geom& g = a.g;
  const XRows<N, DA> rows(g);
  const int grp = threadIdx.x / G, tl = threadIdx.x % G;
  const int MW = rows.Mx() * W;
  xf_twiddles<T, N, W>(tws, a.tw);
  pdl_wait();
  pdl_trigger();
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = tile / nzt, z0 = (tile % nzt) * W;
    const long long cbase = (long long)j * g.Mzp + z0;
    if (grp < 3) {
      Stage0<T, N, W, G> s0;
      const V2<T>* src = a.t3 + grp * a.t_c + cbase;
      const uint32_t sx = (uint32_t)a.t_x * (uint32_t)sizeof(V2<T>);
      s0.load(tl, [&](int b, int lo, int col) {
        return elem(src, (uint32_t)(b + lo) * sx + col * (uint32_t)sizeof(V2<T>));
      });
      cta_sync();  // the previous tile has left X and F (and the twiddles are there)
      s0.template store<false>(tl, X + grp * XT::SLOTS);
      group_sync<G>(grp);
      V2<T>* f = F + grp * MW;
      xf_stage1<T, N, W, G, false>(tl, X + grp * XT::SLOTS, tws, [&](int b, int lo, int col, V2<T> v, V2<T>*) {
        const int row = rows.row(b, lo, XT::R0);
        if (row >= 0) f[row * W + col] = v;
      });
    } else {
      // meanwhile the other groups pull the state rows of the epilogue into L2
      const int nq = a.stage <= 1 ? 3 : 9;  // (array, component): u | s, acc, u
      for (int q = 0; q < nq; ++q) {
        const V2<T>* arr = q < 3 ? (a.stage <= 1 ? a.u : a.s) : (q < 6 ? a.acc : a.u);
        const V2<T>* base = arr + (q % 3) * a.c_c + cbase;
        for (int i = threadIdx.x - 3 * G; i < rows.Mx(); i += 2 * G)
          prefetch_l2(base + (long long)i * a.c_x);
      }
      cta_sync();
    }
    __syncthreads();  // F complete
    const int fy = full_pos(j, g.hy, g.My, g.Ny);
    const T ky = a.k.ky[fy];
    const T cf = (a.forcing == 2 || a.forcing == 3) ? T(a.coef[0]) : T(0);
    double sE = 0.0, sO = 0.0, sB = 0.0;
    const int col = threadIdx.x % W, z = z0 + col;
    const bool zok = z < g.Mz;
    const T kz = zok ? __ldg(a.k.kz + z) : T(0);
    const uint32_t cx = (uint32_t)a.c_x * (uint32_t)sizeof(V2<T>);
    uint32_t o = (uint32_t)(cbase + col) * (uint32_t)sizeof(V2<T>) + (threadIdx.x / W) * cx;
    for (int i = threadIdx.x / W; i < rows.Mx(); i += NTH / W, o += NTH / W * cx) {
      const int e = i * W + col;
      V2<T> ns[3] = {czero<T>(), czero<T>(), czero<T>()};
      if (zok) {
        V2<T> us[3], ac[3], uu[3];
        p3_load(a, o, us, ac, uu);
        V2<T> du[3] = {F[e], F[MW + e], F[2 * MW + e]};
        const int pos = i < rows.hx() ? i : i + N - rows.Mx();
        p3_point(a, pos, fy, z, ky, kz, cf, o, du, us, ac, uu, ns, sE, sO, sB);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) F[c * MW + e] = ns[c];
    }
    if (a.partial) {
      block_sum3_f64(sE, sO, sB, red);
      if (threadIdx.x == 0) {
        a.partial[3 * tile + 0] = sE;
        a.partial[3 * tile + 1] = sO;
        a.partial[3 * tile + 2] = sB;
      }
    }
    if (a.fuse_p1) {
      __syncthreads();  // the new stage input is complete
      xf_inverse<T, N, W, G, DA>(F, X, tws, j, z0, g, a.k, a.t6, a.t6_c, a.t6_x);
    }
  }
}

template <typename T, int N, int W, int G, int MINB, bool DA>
__global__ void __launch_bounds__(XF_GROUPS* G, MINB) k_p1f(P1Args<T> a, int nzt, int ntiles, int f_off) {
  using XT = XTile<N, W>;
  constexpr int NTH = XF_GROUPS * G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<T>* tws = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* X = tws + XT::TWS;
  V2<T>* F = X + f_off;
  const Geom& g = a.g;
  const XRows<N, DA> rows(g);
  const int MW = rows.Mx() * W;
  xf_twiddles<T, N, W>(tws, a.tw);
  pdl_wait();
  pdl_trigger();
  const int col = threadIdx.x % W;
  const uint32_t cx = (uint32_t)a.s_x * (uint32_t)sizeof(V2<T>);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = tile / nzt, z0 = (tile % nzt) * W;
    const V2<T>* src = a.s + (long long)j * g.Mzp + z0;
    __syncthreads();  // the previous tile has left X
    uint32_t o = col * (uint32_t)sizeof(V2<T>) + (threadIdx.x / W) * cx;
#pragma unroll 2
    for (int i = threadIdx.x / W; i < rows.Mx(); i += NTH / W, o += NTH / W * cx) {
#pragma unroll
      for (int c = 0; c < 3; ++c) F[c * MW + i * W + col] = elem(src + c * a.s_c, o);
    }
    __syncthreads();
    xf_inverse<T, N, W, G, DA>(F, X, tws, j, z0, g, a.k, a.t6, a.t_c, a.t_x);
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

template <typename T> cudaError_t launch_p3f(const P3Args<T>& a, cudaStream_t st) {
  return dispatch_two<T>(a.g, [&](auto nn, auto da) {
    constexpr int N = decltype(nn)::value;
    constexpr bool DA = decltype(da)::value;
    using C = XfCfg<T, N, DA>;
    constexpr auto kernel = k_p3f<T, N, C::W, C::G, C::MINB, DA>;
    static PerDevice ready, cache;
    cudaError_t e = once_per_device(ready, [] { return xf_attr(kernel, xf_smem<T, N, C::W>(N)); });
    if (e != cudaSuccess) return e;
    const int nzt = a.g.Mzp / C::W, ntiles = nzt * a.g.My;
    const size_t smem = xf_smem<T, N, C::W>(a.g.Mx);
    const int grid = resident_grid(kernel, XF_GROUPS * C::G, smem, ntiles, cache);
    return launch_pdl(kernel, grid, XF_GROUPS * C::G, smem, st, a, nzt, ntiles, xf_f_off<N, C::W>(a.g.Mx));
  });
}

template <typename T> cudaError_t launch_p1f(const P1Args<T>& a, cudaStream_t st) {
  return dispatch_two<T>(a.g, [&](auto nn, auto da) {
    constexpr int N = decltype(nn)::value;
    constexpr bool DA = decltype(da)::value;
    using C = XfCfg<T, N, DA>;
    constexpr auto kernel = k_p1f<T, N, C::W, C::G, C::MINB, DA>;
    static PerDevice ready, cache;
    cudaError_t e = once_per_device(ready, [] { return xf_attr(kernel, xf_smem<T, N, C::W>(N)); });
    if (e != cudaSuccess) return e;
    const int nzt = a.g.Mzp / C::W, ntiles = nzt * a.g.My;
    const size_t smem = xf_smem<T, N, C::W>(a.g.Mx);
    const int grid = resident_grid(kernel, XF_GROUPS * C::G, smem, ntiles, cache);
    return launch_pdl(kernel, grid, XF_GROUPS * C::G, smem, st, a, nzt, ntiles, xf_f_off<N, C::W>(a.g.Mx));
  });
}

template cudaError_t launch_p3f<float>(const P3Args<float>&, cudaStream_t);
template cudaError_t launch_p3f<double>(const P3Args<double>&, cudaStream_t);
template cudaError_t launch_p1f<float>(const P1Args<float>&, cudaStream_t);
template cudaError_t launch_p1f<double>(const P1Args<double>&, cudaStream_t);

}  // namespace hit
