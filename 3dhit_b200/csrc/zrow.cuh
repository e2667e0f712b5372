// Row transforms along z shared by the z kernels (k_z.cu, k_zadj.cu): the c2r
// pre-processing and r2c post-processing of half-length rows, the row layout
// and twiddle tables of the CTA-per-row-group kernels, and the dispatch on the
// half length.
#pragma once

#include <type_traits>

#include "fft_core.cuh"
#include "kernels.h"

namespace hit {

constexpr int Z_WAIT = 1 << 22;  // mbarrier polls before a TMA wait gives up

template <int H> __host__ __device__ constexpr int z_rows_per_block() {
  return (512 / H) > 32 ? 32 : (512 / H < 1 ? 1 : 512 / H);
}
// threads per block: one per last-stage butterfly of the 3*RB forward rows
template <int H> __host__ __device__ constexpr int z_threads() {
  return ((3 * z_rows_per_block<H>() * (H / fft16_radix(H, fft16_nstages(H) - 1)) + 31) / 32 * 32) < 96
             ? 96
             : ((3 * z_rows_per_block<H>() * (H / fft16_radix(H, fft16_nstages(H) - 1)) + 31) / 32 * 32);
}
// rows of Mzp entries are at most this long (Mzp <= round_up(H+1, 8))
template <int H> __host__ __device__ constexpr int z_row_cap() { return (H + 1 + 7) / 8 * 8; }

// conj-paired pre-processing of one c2r row element k in [0, H).
template <typename T>
__device__ __forceinline__ V2<T> c2r_pre(const V2<T>* row, int k, int H, int Mz, const V2<T>* twz) {
  V2<T> X = k < Mz ? row[k] : czero<T>();
  const int kk = H - k;  // in [1, H]
  V2<T> Y = kk < Mz ? row[kk] : czero<T>();
  if (k == 0) {
    X.y = T(0);
    Y.y = T(0);  // kk == H: Nyquist
  }
  Y.y = -Y.y;  // conj X[H-k]
  const V2<T> s = cadd(X, Y), d = csub(X, Y);
  V2<T> w = twz[k];
  w.y = -w.y;  // e^{+2 pi i k / Nz}
  return cadd(s, cmul_i(cmul(w, d)));
}

// r2c post-processing: output bin k in [0, H] from Z (length H), Z[i] = z(i).
// HALVE = false returns twice the bin (for callers that fold the 1/2 into
// their input scale).
template <typename T, bool HALVE = true, class ZF>
__device__ __forceinline__ V2<T> r2c_post(ZF&& z, int k, int H, const V2<T>* twz) {
  const V2<T> a = z(k == H ? 0 : k);
  V2<T> b = z(k == 0 ? 0 : H - k);
  b.y = -b.y;
  V2<T> E = cadd(a, b), O = cmul_mi(csub(a, b));
  if constexpr (HALVE) {
    E = cscale(E, T(0.5));
    O = cscale(O, T(0.5));
  }
  const V2<T> w = twz[k];  // e^{-2 pi i k / Nz}
  return cadd(E, cmul(w, O));
}

// Shared twiddles of the z kernels: the FFT stage tables (length H, radix-16
// plan) followed by exp(-2 pi i k / Nz) for k in [0, H].
template <int H> __host__ __device__ constexpr int z_tw_slots() { return (tw_size<true>(H) + H + 1 + 1) / 2 * 2; }
// (an even slot count keeps whatever follows the tables 16-byte aligned)
template <typename T, int H, int NTH>
__device__ __forceinline__ void fill_z_twiddles(V2<T>* tws, const V2<T>* __restrict__ tw) {
  fill_stage_twiddles<T, H, true, NTH>(tws, tw);
  V2<T>* twz = tws + tw_size<true>(H);
  for (int k = threadIdx.x; k <= H; k += NTH) twz[k] = tw[k * (TWN / (2 * H))];
  __syncthreads();
}

// DA: the dealiased layout, Mz = Nz/3 + 1 and Mzp = Mz rounded up to 8 as
// compile-time constants, so the bounds of the pre-processing loads and of
// the outputs fold into each value's position range (known-zero inputs are
// not loaded, outputs past the row are not formed).
template <int H> constexpr int zw_da_mz() { return (2 * H) / 3 + 1; }

template <typename F> cudaError_t dispatch_half(int H, F&& f) {
  switch (H) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 16: return f(std::integral_constant<int, 16>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    case 256: return f(std::integral_constant<int, 256>{});
    case 512: return f(std::integral_constant<int, 512>{});
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hit
