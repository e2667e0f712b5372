// x-axis ends of the fused RHS transpose (columns with xf_columns): the
// field-parallel transforms of xfield.cuh around the pointwise algebra of
// k_adjoint.cu.
//   k_adjx1: loads the state u and the cotangent v of a tile, forms pv =
//            project(dealias(v)) and the six float64 sums of the forcing
//            transpose, and runs the x-inverses of u, om = 1j k x u and pv / w
//            (eight transforms, nine fields out);
//   k_adjx2: x-forward of the six products, the cotangent of u, and the
//            algebra of the RK4 step's transpose on it.
// With the z pass in between (k_zadj.cu) a transpose of the RHS is five passes
// over memory.  As separate transforms and pointwise passes over the reference
// layout (k_adj_sums, k_adj_prep, three passes each way, k_adj_cross,
// k_adj_combine, axpys) it was sixteen launches and took 0.50 ms at 128^3.  On
// the dealiased layout the inverse passes carry only the 2/3 box: u is zero
// outside it, and pv always is.
#include "adj_math.cuh"
#include "xfield.cuh"

namespace hit {

template <typename T, int N, int W, int G, int MINB, bool DA>
__global__ void __launch_bounds__(XF_GROUPS* G, MINB) k_adjx1(AdjX1Args<T> a, int nzt, int ntiles) {
  using XT = XTile<N, W>;
  constexpr int NTH = XF_GROUPS * G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[96];
  V2<T>* tws = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* X = tws + XT::TWS;       // five exchange tiles
  V2<T>* F = X + 5 * XT::SLOTS;   // u, then pv / w: 2 x 3 x Mx x W
  const Geom& g = a.gs;
  const XRows<N, DA> rows(g);
  const int MW = rows.Mx() * W;
  const int grp = threadIdx.x / G, tl = threadIdx.x % G;
  const int col = threadIdx.x % W;
  double s[6] = {0, 0, 0, 0, 0, 0};
  xf_twiddles<T, N, W>(tws, a.tw);
  pdl_wait();
  pdl_trigger();
  constexpr uint32_t ES = sizeof(V2<T>);
  const uint32_t cx = (uint32_t)a.c_x * ES, vx = (uint32_t)g.Ny * (uint32_t)a.v_p * ES;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = tile / nzt, z0 = (tile % nzt) * W, z = z0 + col;
    const int fy = full_pos(j, g.hy, g.My, g.Ny);
    const bool zok = z < g.Mz;
    const T ky = a.k.ky[fy], kz = zok ? a.k.kz[z] : T(0);
    const int w = herm_weight(g, z);
    const T iw = T(1) / (T)w;  // 1 or 1/2: exact
    const uint32_t ub = ((uint32_t)j * (uint32_t)g.Mzp + z) * ES, vb = ((uint32_t)fy * (uint32_t)a.v_p + z) * ES;
    __syncthreads();  // the previous tile has left X and F
#pragma unroll 2
    for (int i = threadIdx.x / W; i < rows.Mx(); i += NTH / W) {
      V2<T> u[3] = {czero<T>(), czero<T>(), czero<T>()}, pv[3] = {czero<T>(), czero<T>(), czero<T>()};
      if (zok) {
        const int fx = i < rows.hx() ? i : i + N - rows.Mx();
        V2<T> v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          u[c] = elem(a.u + c * a.c_c, ub + (uint32_t)i * cx);
          v[c] = cscale(elem(a.v + c * a.v_c, vb + (uint32_t)fx * vx), a.vscale);
          pv[c] = v[c];
        }
        Mode<T> d;
        d.kx = __ldg(a.k.kx + fx);
        d.ky = ky;
        d.kz = kz;
        d.k2 = k2_of(d.kx, ky, kz);
        d.ik2 = inv_k2_of(d.k2);
        d.w = w;
        d.keep = DA ? (fx | fy | z) != 0 : in_dealias(g, fx, fy, z);
        proj_mask(d, pv);
        const double pu = re_dot3<T>(pv, u), u2 = re_dot3<T>(u, u), wu2 = w * u2;
        const bool band = a.kmin2 <= d.k2 && d.k2 <= a.kmax2;
        s[0] += pu;
        s[2] += (double)d.k2 * re_dot3<T>(v, u);
        s[3] += wu2;
        s[4] += (double)d.k2 * wu2;
        if (band) {
          s[1] += pu;
          s[5] += wu2;
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        F[c * MW + i * W + col] = u[c];
        F[(3 + c) * MW + i * W + col] = cscale(pv[c], iw);
      }
    }
    __syncthreads();
    xf_inverse<T, N, W, G, DA>(F, X, tws, j, z0, g, a.k, a.t9, a.t_c, a.t_x);
    __syncthreads();  // X is read
    if (grp < 3) {
      Stage0<T, N, W, G> s0;
      const V2<T>* f = F + (3 + grp) * MW;
      s0.load(tl, [&](int b, int lo, int cc) {
        const int row = rows.row(b, lo, XT::R1);
        return row >= 0 ? f[row * W + cc] : czero<T>();
      });
      V2<T>* x = X + grp * XT::SLOTS;
      s0.template store<true>(tl, x);
      group_sync<G>(grp);
      V2<T>* out = a.t9 + (6 + grp) * a.t_c + (long long)j * g.Mzp + z0;
      const uint32_t sx = (uint32_t)a.t_x * ES;
      xf_stage1<T, N, W, G, true>(tl, x, tws, [&](int b, int lo, int cc, V2<T> v, V2<T>*) {
        elem(out, (uint32_t)(b + lo) * sx + (uint32_t)cc * ES) = v;
      });
    }
  }
  block_sum3_f64(s[0], s[1], s[2], red);
  if (threadIdx.x == 0) {
    a.partial[6 * blockIdx.x + 0] = s[0];
    a.partial[6 * blockIdx.x + 1] = s[1];
    a.partial[6 * blockIdx.x + 2] = s[2];
  }
  block_sum3_f64(s[3], s[4], s[5], red);
  if (threadIdx.x == 0) {
    a.partial[6 * blockIdx.x + 3] = s[3];
    a.partial[6 * blockIdx.x + 4] = s[4];
    a.partial[6 * blockIdx.x + 5] = s[5];
  }
}

constexpr int XA_GROUPS = 6;

template <typename T, int N, int W, int G, int MINB>
__global__ void __launch_bounds__(XA_GROUPS* G, MINB) k_adjx2(AdjX2Args<T> a, int nzt, int ntiles) {
  using XT = XTile<N, W>;
  constexpr int NTH = XA_GROUPS * G;
  static_assert(NTH % W == 0, "a thread keeps its column");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<T>* tws = reinterpret_cast<V2<T>*>(smem_raw);
  V2<T>* X = tws + XT::TWS;  // six exchange tiles
  const Geom& g = a.g;
  const int grp = threadIdx.x / G, tl = threadIdx.x % G;
  const int col = threadIdx.x % W;
  xf_twiddles<T, N, W>(tws, a.tw);
  pdl_wait();
  pdl_trigger();
  constexpr uint32_t ES = sizeof(V2<T>);
  // cotangents and products share the padded general layout
  const long long r_c = (long long)N * g.Ny * g.Mzp;
  const uint32_t rx = (uint32_t)g.Ny * (uint32_t)g.Mzp * ES, cx = (uint32_t)a.c_x * ES;
  const double* sc = a.scal;
  const T a_all = (T)sc[0], a_band = (T)sc[1], c_w = (T)sc[2], c_wk2 = (T)sc[3], c_wb = (T)sc[4];
  T nf = T(0);  // sum of 0 v over the modes that the state does not store: NaN where v is not finite
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int j = tile / nzt, z0 = (tile % nzt) * W, z = z0 + col;
    const uint32_t tb = ((uint32_t)j * (uint32_t)g.Mzp + z0) * ES;
    {
      Stage0<T, N, W, G> s0;
      const V2<T>* src = a.r6 + grp * r_c;
      s0.load(tl, [&](int b, int lo, int cc) { return elem(src, tb + (uint32_t)(b + lo) * rx + (uint32_t)cc * ES); });
      __syncthreads();  // the previous tile has left X (and the twiddles are there)
      s0.template store<false>(tl, X + grp * XT::SLOTS);
      group_sync<G>(grp);
      xf_stage1<T, N, W, G, false>(tl, X + grp * XT::SLOTS, tws, [&](int, int, int, V2<T> v, V2<T>* slot) { *slot = v; });
    }
    __syncthreads();
    const bool zok = z < g.Nzh;
    const T ky = a.k.ky[j], kz = zok ? a.k.kz[z] : T(0);
    const int w = herm_weight(g, z);
    // the state's row j and column z, where it is stored
    const int uj = compact_row(j, a.gs.hy, a.gs.My, a.gs.Ny);
    const bool in_yz = uj >= 0 && z < a.gs.Mz;
    const uint32_t ub = ((uint32_t)(uj < 0 ? 0 : uj) * (uint32_t)a.gs.Mzp + z) * ES;
    uint32_t o = tb + (uint32_t)col * ES + (threadIdx.x / W) * rx;
    if (zok) {
      for (int pos = threadIdx.x / W; pos < N; pos += NTH / W, o += NTH / W * rx) {
        V2<T> u[3], v[3], pv[3], bi[3], ac[3], fb[3];
        const int row = compact_row(pos, a.gs.hx, a.gs.Mx, N);
        const bool in = in_yz && row >= 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          u[c] = in ? elem(a.u + c * a.c_c, ub + (uint32_t)row * cx) : czero<T>();
          v[c] = cscale(elem(a.v + c * r_c, o), a.vscale);
          if (a.mode >= 2) bi[c] = elem(a.ubin + c * r_c, o);
          if (a.mode >= 1 && a.mode <= 3) ac[c] = elem((const V2<T>*)a.acc + c * r_c, o);
          if (a.fb && !a.fb_first) fb[c] = elem((const V2<T>*)a.fb + c * r_c, o);
          pv[c] = v[c];
          if (!in) nf += T(0) * v[c].x + T(0) * v[c].y;
        }
        Mode<T> d;
        d.kx = __ldg(a.k.kx + pos);
        d.ky = ky;
        d.kz = kz;
        d.k2 = k2_of(d.kx, ky, kz);
        d.ik2 = inv_k2_of(d.k2);
        d.w = w;
        d.keep = in_dealias(g, pos, j, z);
        proj_mask(d, pv);
        const V2<T>* p = X + XT::at(pos, col);
        V2<T> B[3] = {p[3 * XT::SLOTS], p[4 * XT::SLOTS], p[5 * XT::SLOTS]}, cb[3];
        curl_of(d, B, cb);
        const bool band = a.kmin2 <= d.k2 && d.k2 <= a.kmax2;
        const T ap = a_all + (band ? a_band : T(0));
        const T cu = (T)w * (c_w + d.k2 * c_wk2 + (band ? c_wb : T(0)));
        const T nk2 = a.nu * d.k2;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          V2<T> sb;
          sb.x = -nk2 * v[c].x + ap * pv[c].x + cu * u[c].x;
          sb.y = -nk2 * v[c].y + ap * pv[c].y + cu * u[c].y;
          sb = cadd(sb, cscale(cadd(p[c * XT::SLOTS], cb[c]), (T)w));
          if (a.mode == 0) elem(a.out + c * r_c, o) = sb;
          else if (a.mode == 1) elem(a.out + c * r_c, o) = cadd(ac[c], sb);
          else {
            elem(a.acc + c * r_c, o) = cadd(a.mode == 4 ? bi[c] : ac[c], sb);
            elem(a.kb + c * r_c, o) = cadd(cscale(bi[c], a.c1), cscale(sb, a.c2));
          }
          if (a.fb) elem(a.fb + c * r_c, o) = a.fb_first ? v[c] : cadd(v[c], fb[c]);
        }
      }
    }
  }
  // nu's cotangent is -sum k2 Re(conj(v) u) over all modes; k_adjx1 sums those of
  // the box, the others add 0 v
  if (nf != T(0)) atomicAdd(a.pct, (double)nf);
}

// One warp per sum: Kahan over the blocks' partials (lane stride 32), a fixed
// shuffle tree, then the scalars by one thread.
__global__ void __launch_bounds__(192) k_adj_scal(const double* partial, int nblocks, AdjCoefArgs a) {
  __shared__ double sums[6];
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
  double s = 0.0, c = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblocks; b += 32) {
    const double y = partial[6LL * b + v] - c, t = s + y;
    c = (t - s) - y;
    s = t;
  }
  s -= c;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sums[v] = s;
  __syncthreads();
  if (threadIdx.x == 0) adj_coef(a, sums);
}

cudaError_t launch_adj_scal(const double* partial, int nblocks, const AdjCoefArgs& a, cudaStream_t st) {
  return launch_pdl(k_adj_scal, 1, 192, 0, st, partial, nblocks, a);
}

template <typename T> cudaError_t launch_adj_x1(const AdjX1Args<T>& a, int* nblocks, cudaStream_t st) {
  return dispatch_two<T>(a.gs, [&](auto nn, auto da) {
    constexpr int N = decltype(nn)::value;
    constexpr bool DA = decltype(da)::value;
    using C = XfCfg<T, N, DA>;
    using XT = XTile<N, C::W>;
    constexpr int MINB = N == 256 ? 1 : 2;
    constexpr auto kernel = k_adjx1<T, N, C::W, C::G, MINB, DA>;
    const size_t smem = sizeof(V2<T>) * (size_t)(XT::TWS + 5 * XT::SLOTS + 6 * a.gs.Mx * C::W);
    static PerDevice ready, cache;
    cudaError_t e = once_per_device(ready, [&] { return xf_attr(kernel, smem); });
    if (e != cudaSuccess) return e;
    const int nzt = a.gs.Mzp / C::W, ntiles = nzt * a.gs.My;
    *nblocks = resident_grid(kernel, XF_GROUPS * C::G, smem, ntiles, cache);
    return launch_pdl(kernel, *nblocks, XF_GROUPS * C::G, smem, st, a, nzt, ntiles);
  });
}

template <typename T> cudaError_t launch_adj_x2(const AdjX2Args<T>& a, cudaStream_t st) {
  return dispatch_two<T>(a.g, [&](auto nn, auto) {
    constexpr int N = decltype(nn)::value;
    using C = XfCfg<T, N, true>;
    using XT = XTile<N, C::W>;
    constexpr int MINB = N == 256 || (N == 128 && sizeof(T) == 8) ? 1 : 2;
    constexpr auto kernel = k_adjx2<T, N, C::W, C::G, MINB>;
    const size_t smem = sizeof(V2<T>) * (size_t)(XT::TWS + XA_GROUPS * XT::SLOTS);
    static PerDevice ready, cache;
    cudaError_t e = once_per_device(ready, [&] { return xf_attr(kernel, smem); });
    if (e != cudaSuccess) return e;
    const int nzt = a.g.Mzp / C::W, ntiles = nzt * a.g.Ny;
    const int grid = resident_grid(kernel, XA_GROUPS * C::G, smem, ntiles, cache);
    return launch_pdl(kernel, grid, XA_GROUPS * C::G, smem, st, a, nzt, ntiles);
  });
}

template cudaError_t launch_adj_x1<float>(const AdjX1Args<float>&, int*, cudaStream_t);
template cudaError_t launch_adj_x1<double>(const AdjX1Args<double>&, int*, cudaStream_t);
template cudaError_t launch_adj_x2<float>(const AdjX2Args<float>&, cudaStream_t);
template cudaError_t launch_adj_x2<double>(const AdjX2Args<double>&, cudaStream_t);

}  // namespace hit
