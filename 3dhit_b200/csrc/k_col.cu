// Column FFTs along a strided axis, short lengths (col_pass in kernels.h: the y
// passes of the RHS and the x and y passes of the 3-D transforms), two stages
// per transform.
//
// A group of G threads owns one tile (all N rows along the axis times W
// contiguous z columns): each thread loads the inputs of its first-stage
// butterflies straight from global memory into registers (up to 16 rows in
// flight per thread), the stages meet in one shared-memory exchange ordered by
// the group's own barrier, and the second stage stores straight to global
// memory.  A CTA holds several groups that walk their tiles independently: no
// CTA barrier in the loop, no staging copy, no alignment requirement on rows.
// k_axis works on one tile per CTA, whose 256 threads have no butterfly at all
// in most short stages.  Six y-inverse fields, k_axis -> k_col: 512 x 16 x 512
// 86 -> 27 us, 512 x 32 x 512 107 -> 58, 512 x 64 x 512 125 -> 107, 64 points in
// 128 x 64 x 256 19 -> 15.  At 128 and 256 points TMA staging (k_axis2) is
// faster (256^3: 82 against 124 us), whatever the number of loads in flight here
// (next tile's loads held in registers: 127).
#include "xfield.cuh"

namespace hit {

constexpr int COL_THREADS = 256;
template <typename T, int N> struct ColCfg {
  static constexpr int W = tile_w<T>(N);
  static constexpr int B = Two<N>::R1 * W;  // first-stage butterflies of a tile
  static constexpr int G = B <= 32 ? 32 : (B >= 128 && N == 256 ? 128 : 64);
  static constexpr int GP = COL_THREADS / G;  // groups (tiles) per CTA
};

// ROWS: the compact side stores 0 any rows, 1 the 2/3 box, 2 all of them (M = N)
template <typename T, int N, bool INV, int ROWS>
__global__ void __launch_bounds__(COL_THREADS, sizeof(T) == 4 ? 4 : 2) k_col(AxisArgs<T> a, int nzt, int no, int ntiles) {
  using C = ColCfg<T, N>;
  constexpr int W = C::W, G = C::G;
  using XT = XTile<N, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<T>* tws = reinterpret_cast<V2<T>*>(smem_raw);
  const int grp = threadIdx.x / G, tl = threadIdx.x % G;
  V2<T>* x = tws + XT::TWS + grp * XT::SLOTS;
  xf_twiddles<T, N, W>(tws, a.tw);
  const ColRows<N, ROWS == 1> rows{INV ? a.hin : a.hout, INV ? a.Min : a.Mout};
  pdl_wait();
  if (ROWS == 1) pdl_trigger();  // (other layouts: 64^3 step 121 us with it, 111 without)
  __syncthreads();  // the twiddles
  constexpr uint32_t ES = sizeof(V2<T>);
  const uint32_t sa = (uint32_t)a.s_a * ES, da = (uint32_t)a.d_a * ES;
  for (int tile = blockIdx.x * C::GP + grp; tile < ntiles; tile += gridDim.x * C::GP) {
    const int zt = tile % nzt, q = tile / nzt, o = q % no, c = q / no;
    const int z0 = zt * W;
    const V2<T>* src = a.src + (long long)c * a.s_c + (long long)o * a.s_o + z0;
    V2<T>* dst = a.dst + (long long)c * a.d_c + (long long)o * a.d_o + z0;
    const int nc = a.nz - z0;  // valid columns of the tile
    Stage0<T, N, W, G> s0;
    s0.load(tl, [&](int b, int lo, int col) {
      const int row = (INV && ROWS != 2) ? rows.row(b, lo, XT::R1) : lo + b;
      return row >= 0 && col < nc ? elem(src, (uint32_t)row * sa + (uint32_t)col * ES) : czero<T>();
    });
    group_sync<G>(grp);  // the group has left its exchange tile
    s0.template store<INV>(tl, x);
    group_sync<G>(grp);
    xf_stage1<T, N, W, G, INV>(tl, x, tws, [&](int b, int lo, int col, V2<T> v, V2<T>*) {
      const int row = (!INV && ROWS != 2) ? rows.row(b, lo, XT::R0) : lo + b;
      if (row >= 0 && col < nc) elem(dst, (uint32_t)row * da + (uint32_t)col * ES) = v;
    });
  }
}

template <typename T, int N, bool INV, int ROWS>
cudaError_t launch_col_v(const AxisArgs<T>& a, int nzt, int no, int nc, cudaStream_t st) {
  using C = ColCfg<T, N>;
  using XT = XTile<N, C::W>;
  constexpr size_t smem = sizeof(V2<T>) * (size_t)(XT::TWS + C::GP * XT::SLOTS);
  constexpr auto kernel = k_col<T, N, INV, ROWS>;
  static PerDevice ready, cache;
  cudaError_t e = once_per_device(ready, [] { return xf_attr(kernel, smem); });
  if (e != cudaSuccess) return e;
  const long long ntiles = (long long)nzt * no * nc;
  const int grid = resident_grid(kernel, COL_THREADS, smem, (ntiles + C::GP - 1) / C::GP, cache);
  return launch_pdl(kernel, grid, COL_THREADS, smem, st, a, nzt, no, (int)ntiles);
}

template <typename T>
cudaError_t launch_col(int N, bool inv, const AxisArgs<T>& a, int nzt, int no, int nc, cudaStream_t st) {
  if ((inv ? a.Mout : a.Min) != N) return cudaErrorInvalidValue;  // the full side is all N rows
  auto go = [&](auto nn) {
    constexpr int NN = decltype(nn)::value;
    const int M = inv ? a.Min : a.Mout, h = inv ? a.hin : a.hout;
    const int rows = M == NN ? 2 : (M == 2 * (NN / 3) + 1 && h == NN / 3 + 1 ? 1 : 0);
    if (inv)
      return rows == 2   ? launch_col_v<T, NN, true, 2>(a, nzt, no, nc, st)
             : rows == 1 ? launch_col_v<T, NN, true, 1>(a, nzt, no, nc, st)
                         : launch_col_v<T, NN, true, 0>(a, nzt, no, nc, st);
    return rows == 2   ? launch_col_v<T, NN, false, 2>(a, nzt, no, nc, st)
           : rows == 1 ? launch_col_v<T, NN, false, 1>(a, nzt, no, nc, st)
                       : launch_col_v<T, NN, false, 0>(a, nzt, no, nc, st);
  };
  switch (N) {
    case 4: return go(std::integral_constant<int, 4>{});
    case 8: return go(std::integral_constant<int, 8>{});
    case 16: return go(std::integral_constant<int, 16>{});
    case 32: return go(std::integral_constant<int, 32>{});
    case 64: return go(std::integral_constant<int, 64>{});
    case 128: return go(std::integral_constant<int, 128>{});
    case 256: return go(std::integral_constant<int, 256>{});
    default: return cudaErrorInvalidValue;
  }
}

template cudaError_t launch_col<float>(int, bool, const AxisArgs<float>&, int, int, int, cudaStream_t);
template cudaError_t launch_col<double>(int, bool, const AxisArgs<double>&, int, int, int, cudaStream_t);

}  // namespace hit
