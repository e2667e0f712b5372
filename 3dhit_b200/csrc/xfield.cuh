// Field-parallel column transforms along x (columns with xf_columns): the
// two-stage transforms of k_xfield.cu and k_xadj.cu, their shared-memory layout
// and the launch configuration.
#pragma once

#include <type_traits>

#include "fft_core.cuh"
#include "kernels.h"
#include "p3_epilogue.cuh"

namespace hit {

// Radices of the two stages.
template <int N> struct Two {
  static constexpr int L = ilog2(N);
  static constexpr int R0 = 1 << (L / 2), R1 = N / R0;  // R0 <= R1 <= 32
  static_assert(N >= 4 && R1 <= 32, "two-stage columns");
};

// Shared-memory layout of a field's exchange tile: slot (pos + pos / R0) W +
// col.  A pad row after every R0 positions lets the stage-0 stores (positions
// R0 b + r of consecutive b) and the stage-1 loads (b + R0 r) of a half warp
// hit both halves of the banks.
template <int N, int W> struct XTile {
  static constexpr int R0 = Two<N>::R0, R1 = Two<N>::R1;
  static constexpr int SLOTS = (N + N / R0) * W;
  static constexpr int TWS = ((R1 - 1) * R0 + 1) / 2 * 2;
  static __device__ __forceinline__ int at(int pos, int col) { return (pos + pos / R0) * W + col; }
};

constexpr int XF_GROUPS = 5;

template <int G> __device__ __forceinline__ void group_sync(int g) {
  if constexpr (G == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(G) : "memory");
}

// The CTA barrier, for code where the groups are on different paths.
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

// Stage-1 twiddles w_N^{r k} at slot (r - 1) R0 + k.
template <typename T, int N, int W>
__device__ __forceinline__ void xf_twiddles(V2<T>* tws, const V2<T>* __restrict__ tw) {
  using X = XTile<N, W>;
  for (int e = threadIdx.x; e < (X::R1 - 1) * X::R0; e += blockDim.x)
    tws[e] = tw[(e / X::R0 + 1) * (e % X::R0) * (TWN / N)];
}

// Stored rows of one side: compile-time when they are the 2/3 box (DA), so that the
// bounds of a butterfly's positions fold into constants.
template <int N, bool DA> struct ColRows {
  int h_, M_;
  __device__ __forceinline__ int h() const { return DA ? N / 3 + 1 : h_; }
  __device__ __forceinline__ int M() const { return DA ? 2 * (N / 3) + 1 : M_; }
  // stored row of position lo + b, b in [0, nb) (nb and lo constants), or -1
  __device__ __forceinline__ int row(int b, int lo, int nb) const {
    const int off = N - M();
    if (DA && lo + nb <= h()) return lo + b;
    if (DA && lo >= h() + off) return lo + b - off;
    if (DA && lo >= h() && lo + nb <= h() + off) return -1;
    const int pos = lo + b;
    return pos < h() ? pos : (pos >= h() + off ? pos - off : -1);
  }
};

// The stored x rows.
template <int N, bool DA> struct XRows : ColRows<N, DA> {
  __device__ __forceinline__ explicit XRows(const Geom& g) : ColRows<N, DA>{g.hx, g.Mx} {}
  __device__ __forceinline__ int hx() const { return this->h(); }
  __device__ __forceinline__ int Mx() const { return this->M(); }
};

// Stage 0 of a group's transform in two parts: the loads of all its
// butterflies (positions b + r R1: ld(b, r R1, col)), and the butterflies with
// their stores into the exchange tile.
template <typename T, int N, int W, int G> struct Stage0 {
  using X = XTile<N, W>;
  static constexpr int R = X::R0, NB = X::R1, TOTAL = NB * W, CNT = (TOTAL + G - 1) / G;
  V2<T> v[CNT][R];
  template <class LD> __device__ __forceinline__ void load(int tl, LD&& ld) {
#pragma unroll
    for (int c = 0; c < CNT; ++c) {
      const int t = tl + c * G;
      if (TOTAL % G == 0 || t < TOTAL) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[c][r] = ld(t / W, r * NB, t % W);
      }
    }
  }
  template <bool INV> __device__ __forceinline__ void store(int tl, V2<T>* x) {
#pragma unroll
    for (int c = 0; c < CNT; ++c) {
      const int t = tl + c * G;
      if (TOTAL % G == 0 || t < TOTAL) {
        DFT<R, INV, V2<T>>::run(v[c]);
        V2<T>* p = x + (t / W) * (R + 1) * W + t % W;
#pragma unroll
        for (int r = 0; r < R; ++r) p[r * W] = v[c][r];
      }
    }
  }
};

// Stage 1: butterfly b takes positions b + r R0 and gives the same positions,
// st(b, r R0, col, value, slot pointer).
template <typename T, int N, int W, int G, bool INV, class ST>
__device__ __forceinline__ void xf_stage1(int tl, V2<T>* x, const V2<T>* tws, ST&& st) {
  using X = XTile<N, W>;
  constexpr int R = X::R1, NB = X::R0, TOTAL = NB * W, CNT = (TOTAL + G - 1) / G;
#pragma unroll
  for (int c = 0; c < CNT; ++c) {
    const int t = tl + c * G;
    if (TOTAL % G == 0 || t < TOTAL) {
      const int b = t / W, col = t % W;
      V2<T>* p = x + b * W + col;
      V2<T> v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = p[r * (NB + 1) * W];
#pragma unroll
      for (int r = 1; r < R; ++r) {
        V2<T> w = tws[(r - 1) * NB + b];
        if (INV) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
      DFT<R, INV, V2<T>>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) st(b, r * NB, col, v[r], p + r * (NB + 1) * W);
    }
  }
}

// x-inverse of the tile's field F (3 x Mx x W compact rows in shared memory)
// and of w = i k x u, as p1_body: five transforms, one per group.  F may
// overlap the exchange tiles X (every thread has loaded its stage-0 inputs
// before any store).  The caller synchronises after F is written; returns
// after the block's last read of X has been issued (not synchronised).
template <typename T, int N, int W, int G, bool DA>
__device__ __forceinline__ void xf_inverse(const V2<T>* F, V2<T>* X, const V2<T>* tws, int j, int z0, const Geom& g,
                                           const KTab<T>& kt, V2<T>* t6, long long t_c, long long t_x) {
  using XT = XTile<N, W>;
  const XRows<N, DA> rows(g);
  const int grp = threadIdx.x / G, tl = threadIdx.x % G;
  V2<T>* x = X + grp * XT::SLOTS;
  {
    Stage0<T, N, W, G> s0;
    const int comp = grp < 3 ? grp : grp - 2;  // u_x, kx u_y, kx u_z, u_y, u_z
    const bool kxs = grp == 1 || grp == 2;
    const V2<T>* f = F + comp * rows.Mx() * W;
    s0.load(tl, [&](int b, int lo, int col) {
      const int row = rows.row(b, lo, XT::R1);
      return row >= 0 ? f[row * W + col] : czero<T>();
    });
    if (kxs) {
#pragma unroll
      for (int c = 0; c < s0.CNT; ++c) {
        const int b = (tl + c * G) / W;
        if (s0.TOTAL % G == 0 || tl + c * G < s0.TOTAL) {
#pragma unroll
          for (int r = 0; r < s0.R; ++r) {
            if (!DA || rows.row(0, r * XT::R1, XT::R1) >= 0 || rows.row(XT::R1 - 1, r * XT::R1, XT::R1) >= 0)
              s0.v[c][r] = cscale(s0.v[c][r], __ldg(kt.kx + b + r * XT::R1));
          }
        }
      }
    }
    __syncthreads();  // F is read: X may overwrite it
    s0.template store<true>(tl, x);
  }
  group_sync<G>(grp);
  xf_stage1<T, N, W, G, true>(tl, x, tws, [&](int, int, int, V2<T> v, V2<T>* slot) { *slot = v; });
  __syncthreads();
  const T ky = kt.ky[full_pos(j, g.hy, g.My, g.Ny)];
  V2<T>* out = t6 + (long long)j * g.Mzp + z0;
  constexpr int NTH = XF_GROUPS * G;
  static_assert(NTH % W == 0, "a thread keeps its column");
  const int col = threadIdx.x % W, z = z0 + col;
  const T kz = z < g.Nzh ? kt.kz[z] : T(0);
  // 32-bit byte offsets inside a component (N <= 256 rows of at most 1024 x 520
  // entries: below 4 GB)
  const uint32_t sx = (uint32_t)t_x * (uint32_t)sizeof(V2<T>);
  uint32_t o = (threadIdx.x / W) * sx + col * (uint32_t)sizeof(V2<T>);
#pragma unroll 2
  for (int pos = threadIdx.x / W; pos < N; pos += NTH / W, o += NTH / W * sx) {
    const V2<T>* p = X + XT::at(pos, col);
    const V2<T> ux = p[0], xy = p[XT::SLOTS], xz = p[2 * XT::SLOTS], uy = p[3 * XT::SLOTS], uz = p[4 * XT::SLOTS];
    elem(out, o) = ux;
    elem(out + t_c, o) = uy;
    elem(out + 2 * t_c, o) = uz;
    elem(out + 3 * t_c, o) = cmul_i(csub(cscale(uz, ky), cscale(uy, kz)));
    elem(out + 4 * t_c, o) = cmul_i(csub(cscale(ux, kz), xz));
    elem(out + 5 * t_c, o) = cmul_i(csub(xy, cscale(ux, ky)));
  }
}

// ---------------------------------------------------------------------------
// launch configuration
// ---------------------------------------------------------------------------

// Tile width (64-byte row segments), threads per group and CTAs per SM that
// the register budget is sized for.  x-forward pass at 128 float points, budget
// for 2, 3 and 4 CTAs: general 128^3 66, 70 and 81 us, 2/3 box of 128 x 64 x 256
// 27.4, 27.9 and 28.9; at 64 points 10.7, 10.7 (3) and 12.2 (4), general 18.6, 16.2,
// 16.7; float64 57 us for 2 CTAs, 76 for 3, 63 for 1.
template <typename T, int N, bool DA> struct XfCfg {
  static constexpr int W = xf_tile_w<T>();
  static constexpr int B = Two<N>::R1 * W;  // stage-0 butterflies of a transform
  static constexpr bool F32 = sizeof(T) == 4;
  // float columns of 256 points on the general layout: F does not fit over the
  // exchange tiles, one CTA per SM
  static constexpr bool WIDE = N == 256 && !DA;
  static constexpr int G = B < 64 ? 32 : (WIDE ? B : 64);
  static constexpr int MINB = WIDE ? 1 : (F32 ? (N >= 128 ? 2 : 3) : 2);
};

// Slot offset of F from X: over the exchange tiles of groups 3 and 4 (idle
// while the forward transforms fill F) when it fits there, else behind them.
template <int N, int W> int xf_f_off(int Mx) {
  using XT = XTile<N, W>;
  return 3 * Mx * W <= 2 * XT::SLOTS ? 3 * XT::SLOTS : 5 * XT::SLOTS;
}
template <typename T, int N, int W> size_t xf_smem(int Mx) {
  using XT = XTile<N, W>;
  const int f = xf_f_off<N, W>(Mx);
  return sizeof(V2<T>) * (size_t)(XT::TWS + (f == 3 * XT::SLOTS ? 5 * XT::SLOTS : f + 3 * Mx * W));
}

template <typename K> cudaError_t xf_attr(K kernel, size_t bytes) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

template <int N, typename F> cudaError_t dispatch_da(const Geom& g, F&& f) {
  const std::integral_constant<int, N> n{};
  return g.pruned ? f(n, std::true_type{}) : f(n, std::false_type{});
}
template <typename T, typename F> cudaError_t dispatch_two(const Geom& g, F&& f) {
  if constexpr (xf_columns<T>(256)) {
    if (g.Nx == 256) return dispatch_da<256>(g, f);
  }
  switch (g.Nx) {
    case 4: return dispatch_da<4>(g, f);
    case 8: return dispatch_da<8>(g, f);
    case 16: return dispatch_da<16>(g, f);
    case 32: return dispatch_da<32>(g, f);
    case 64: return dispatch_da<64>(g, f);
    case 128: return dispatch_da<128>(g, f);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hit
