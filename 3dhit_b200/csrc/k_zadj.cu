// z pass of the fused RHS transpose: per (x, y) row, c2r of the nine fields u,
// om = 1j k x u and g (the inverse transforms of pv / w), the products om x g
// and g x u at the grid points, r2c of the six products.  The two forms follow
// k_zwarp (float32 rows of 64 .. 512 points: warp-resident rows, no CTA
// barrier) and k_zcross (every other length and float64: a CTA per row group,
// in-place row transforms in shared memory).  The products never reach memory:
// as c2r, product and r2c passes of their own they moved 30 real fields.
//   128^3 float32: 44.5 + 16.7 + 36.4 us before, see k_xadj.cu for the whole
//   transpose.
#include <algorithm>
#include <type_traits>

#include "fft_core.cuh"
#include "kernels.h"
#include "tma.cuh"
#include "zrow.cuh"
#include "zwarp.cuh"

namespace hit {

__device__ int g_zadj_timeout = 0;  // set when a TMA wait gave up (hit_device_status)
__device__ int g_zadj_wait_limit = Z_WAIT;  // polls of the wait for a row group (hit_set_wait_limit)

cudaError_t set_zadj_wait_limit(int polls) {
  const int v = polls < 0 ? Z_WAIT : polls;
  return cudaMemcpyToSymbol(g_zadj_wait_limit, &v, sizeof(int));
}
cudaError_t take_zadj_timeout(int* flag) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_zadj_timeout, sizeof(int));
  if (e != cudaSuccess) return e;
  *flag = v;
  const int zero = 0;
  return v ? cudaMemcpyToSymbol(g_zadj_timeout, &zero, sizeof(int)) : cudaSuccess;
}

// Generic form: RB rows per group, columns q RB + lr of the shared buffer hold
// field q of row lr (c2r: q < 9; r2c: q < 6).
template <typename T, int H, int RB, int NTZ, int MINB>
__global__ void __launch_bounds__(NTZ, MINB) k_zadj(ZAdjArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using AD = SkewAddr<skew_ld(H)>;
  V2<T>* buf = reinterpret_cast<V2<T>*>(smem_raw);  // 9 RB columns of AD::LD slots
  V2<T>* tws = buf + 9 * RB * AD::LD;
  const V2<T>* twz = tws + tw_size<true>(H);
  constexpr int RS = z_row_cap<H>();
  V2<T>* raw = tws + z_tw_slots<H>();  // staged rows [q RB + lr][RS], zero past Mzp
  fill_z_twiddles<T, H, NTZ>(tws, a.tw);
  const int ngroups = (a.nrows + RB - 1) / RB;
  const int Mzp = a.Mzp;
  for (int e = threadIdx.x; e < 9 * RB * RS; e += NTZ)
    if (e % RS >= Mzp) raw[e] = czero<T>();
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  constexpr int NWARP = NTZ / 32;
  __shared__ __align__(8) uint64_t zbar;
  const uint32_t mb = tma::smem_u32(&zbar);
  if (threadIdx.x == 0) tma::mbar_init(mb, 1);
  tma::fence_async_smem();
  __syncthreads();
  auto prefetch = [&](int grp) {
    if (threadIdx.x < 32) {
      const long long r0 = (long long)grp * RB;
      const int nin = (int)(a.nrows - r0 < RB ? a.nrows - r0 : RB);
      const uint32_t bytes = (uint32_t)(Mzp * sizeof(V2<T>));
      if (threadIdx.x == 0) tma::mbar_expect_tx(mb, 9u * nin * bytes);
      __syncwarp();
      for (int col = threadIdx.x; col < 9 * RB; col += 32) {
        const int q = col / RB, lr = col % RB;
        if (lr < nin) tma::load_bytes(raw + col * RS, a.in + q * a.in_c + (r0 + lr) * Mzp, bytes, mb);
      }
    }
  };
  const int wait_limit = g_zadj_wait_limit;
  pdl_wait();
  pdl_trigger();
  int grp = blockIdx.x;
  if (grp < ngroups) prefetch(grp);
  uint32_t phase = 0;
  for (; grp < ngroups; grp += gridDim.x) {
    const long long row0 = (long long)grp * RB;
    {
      const bool ok = __syncthreads_and(tma::mbar_wait(mb, phase, wait_limit)) != 0;
      phase ^= 1;
      if (!ok) {
        if (threadIdx.x == 0) atomicExch(&g_zadj_timeout, 1);
        tma::mbar_wait(mb, phase ^ 1, Z_WAIT);  // the copies in flight, once more with a limit
        return;
      }
    }
    const int nxt = grp + gridDim.x;
    fft_ip<T, H, 9 * RB, NTZ, AD, true>(
        buf, tws, [&](int k, int col) { return c2r_pre<T>(raw + col * RS, k, H, RS, twz); },
        [&](int m, int col, V2<T> v) { buf[AD::at(m, col)] = v; },
        [&]() {
          if (nxt < ngroups) prefetch(nxt);
        });
    const T s2 = T(0.5) * a.scale * a.scale;  // both inverse normalisations and the r2c 1/2
    fft_ip<T, H, 6 * RB, NTZ, AD, false>(
        buf, tws,
        [&](int m, int col) {
          const int q = col / RB, lr = col % RB, c = q < 3 ? q : q - 3;
          const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;  // (1,2), (2,0), (0,1)
          const int fa = q < 3 ? 3 : 6, fb = q < 3 ? 6 : 0;            // om x g, g x u
          const V2<T> a1 = buf[AD::at(m, (fa + c1) * RB + lr)], a2 = buf[AD::at(m, (fa + c2) * RB + lr)];
          const V2<T> b1 = buf[AD::at(m, (fb + c1) * RB + lr)], b2 = buf[AD::at(m, (fb + c2) * RB + lr)];
          V2<T> n;
          n.x = (a1.x * b2.x - a2.x * b1.x) * s2;
          n.y = (a1.y * b2.y - a2.y * b1.y) * s2;
          return n;
        },
        [&](int k, int col, V2<T> v) { buf[AD::at(k, col)] = v; });
    for (int col = warp; col < 6 * RB; col += NWARP) {
      const int q = col / RB, lr = col % RB;
      if (row0 + lr < a.nrows) {
        V2<T>* out = a.out + q * a.out_c + (row0 + lr) * a.Mzpo;
        for (int k = lane; k < a.Mzpo; k += 32)
          out[k] = k < a.Mzo ? r2c_post<T, false>([&](int i) { return buf[AD::at(i, col)]; }, k, H, twz) : czero<T>();
      }
    }
    __syncthreads();  // buf is rewritten by the next group
  }
}

// Warp-resident form (see k_zwarp).  Per lane and row: u and g are transformed
// first, g x u formed value by value and sent out while both are live, then
// om accumulates om x g as its fields arrive, so at most six fields of eight
// values are held at a time.
constexpr int ZA_WARPS = 4, ZA_MINB = 3;
template <int H, bool DA>
__global__ void __launch_bounds__(ZA_WARPS * 32, ZA_MINB) k_zadjw(ZAdjArgs<float> a) {
  using Z = ZW<H>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[ZA_WARPS];
  float2* tws = reinterpret_cast<float2*>(smem_raw);
  const int Mz = DA ? zw_da_mz<H>() : a.Mz;
  const int Mzp = DA ? (zw_da_mz<H>() + 7) / 8 * 8 : a.Mzp;
  auto below = [](int k, int lo, int hi, int bound) { return hi < bound ? true : (lo >= bound ? false : k < bound); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = lane / Z::LPR, b = lane % Z::LPR;
  ZwMid<H> mid(b);
  float2 wl[7];
  const int stg_slots = 9 * Z::ROWS * Mzp;
  float2* stg = tws + Z::TWS + warp * (stg_slots + Z::ROWS * Z::XS);  // [field][row][Mzp]
  float2* xch = stg + stg_slots + q * Z::XS;
  const float2* twz = tws + Z::TWZ;
  zw_fill_twiddles<H, ZA_WARPS * 32>(tws, a.tw);
  const uint32_t mb = tma::smem_u32(&bars[warp]);
  if (lane == 0) tma::mbar_init(mb, 1);
  tma::fence_async_smem();
  __syncthreads();
  zw_last_twiddles<H>(wl, tws, b);
  mid.load(tws);
  const int wait_limit = g_zadj_wait_limit;
  const long long ngroups = a.nrows / Z::ROWS;
  const long long nwarps = (long long)gridDim.x * ZA_WARPS;
  const uint32_t row_bytes = (uint32_t)(Mzp * sizeof(float2));
  auto prefetch = [&](long long grp) {
    if (lane == 0) tma::mbar_expect_tx(mb, 9u * Z::ROWS * row_bytes);
    __syncwarp();
    for (int i = lane; i < 9 * Z::ROWS; i += 32) {
      const int c = i / Z::ROWS, rr = i % Z::ROWS;
      tma::load_bytes(stg + i * Mzp, a.in + c * a.in_c + (grp * Z::ROWS + rr) * Mzp, row_bytes, mb);
    }
  };
  pdl_wait();
  pdl_trigger();
  long long grp = (long long)blockIdx.x * ZA_WARPS + warp;
  if (grp < ngroups) prefetch(grp);
  uint32_t phase = 0;
  const float s2 = 0.5f * a.scale * a.scale;  // both inverse normalisations and the r2c 1/2
  for (; grp < ngroups; grp += nwarps) {
    {
      const bool ok = __all_sync(0xffffffffu, tma::mbar_wait(mb, phase, wait_limit));
      phase ^= 1;
      if (!ok) {
        if (lane == 0) atomicExch(&g_zadj_timeout, 1);
        tma::mbar_wait(mb, phase ^ 1, Z_WAIT);  // the copies in flight, once more with a limit
        return;
      }
    }
    const float2 wz0 = twz[b];
    // c2r of staged field c
    auto inverse = [&](int c, float2 (&v)[8]) {
      const float2* row = stg + (c * Z::ROWS + q) * Mzp;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int k = b + Z::NB0 * r, kk = H - k;
        float2 X = below(k, Z::NB0 * r, Z::NB0 * r + Z::NB0 - 1, Mz) ? row[k] : make_float2(0.f, 0.f);
        float2 Y = below(kk, H - Z::NB0 * r - Z::NB0 + 1, H - Z::NB0 * r, Mz) ? row[kk] : make_float2(0.f, 0.f);
        if (k == 0) {
          X.y = 0.f;
          Y.y = 0.f;
        }
        Y.y = -Y.y;
        const float2 sm = cadd(X, Y), df = csub(X, Y);
        float2 w = zw_wz(wz0, r);
        w.y = -w.y;
        v[r] = cadd(sm, cmul_i(cmul(w, df)));
      }
      zw_transform<H, true>(v, xch, tws, b, mid, wl);
    };
    // r2c of product c (all H + 1 bins and the row's padding)
    const int partner = q * Z::LPR + ((Z::LPR - b) & (Z::LPR - 1));
    auto forward = [&](int c, float2 (&v)[8]) {
      zw_transform<H, false>(v, xch, tws, b, mid, wl);
      float2* out = a.out + c * a.out_c + (grp * Z::ROWS + q) * a.Mzpo;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        float2 t;
        t.x = __shfl_sync(0xffffffffu, v[7 - r].x, partner);
        t.y = __shfl_sync(0xffffffffu, v[7 - r].y, partner);
        float2 bc = b == 0 ? v[(8 - r) & 7] : t;
        bc.y = -bc.y;
        const float2 E = cadd(v[r], bc), O = cmul_mi(csub(v[r], bc));
        out[b + Z::NB0 * r] = cadd(E, cmul(zw_wz(wz0, r), O));
      }
      for (int k = b; k < a.Mzpo - H; k += Z::LPR) {
        float2 x = make_float2(0.f, 0.f);
        if (k == 0) {
          float2 bc = v[0];
          bc.y = -bc.y;
          x = cadd(cadd(v[0], bc), cmul(twz[H], cmul_mi(csub(v[0], bc))));
        }
        out[H + k] = x;
      }
    };
    float2 p[3][8], g[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) inverse(c, p[c]);
#pragma unroll
    for (int c = 0; c < 3; ++c) inverse(6 + c, g[c]);
    // g x u
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      constexpr int n1[3] = {1, 2, 0}, n2[3] = {2, 0, 1};
      const int c1 = n1[c], c2 = n2[c];
      float2 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float2 m = __fmul2_rn(g[c2][r], make_float2(-p[c1][r].x, -p[c1][r].y));
        v[r] = __fmul2_rn(__ffma2_rn(g[c1][r], p[c2][r], m), make_float2(s2, s2));
      }
      forward(3 + c, v);
    }
    // om x g: n0 = o1 g2 - o2 g1, n1 = o2 g0 - o0 g2, n2 = o0 g1 - o1 g0
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float2 v[8];
      inverse(3 + c, v);
      if (c == 2 && grp + nwarps < ngroups) prefetch(grp + nwarps);  // every lane is past its staged reads
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float2 x = v[r], nx = make_float2(-x.x, -x.y), sc = make_float2(s2, s2);
        if (c == 0) {
          p[1][r] = __fmul2_rn(nx, g[2][r]);
          p[2][r] = __fmul2_rn(x, g[1][r]);
        } else if (c == 1) {
          p[0][r] = __fmul2_rn(x, g[2][r]);
          p[2][r] = __fmul2_rn(__ffma2_rn(nx, g[0][r], p[2][r]), sc);
        } else {
          p[0][r] = __fmul2_rn(__ffma2_rn(nx, g[1][r], p[0][r]), sc);
          p[1][r] = __fmul2_rn(__ffma2_rn(x, g[0][r], p[1][r]), sc);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) forward(c, p[c]);
  }
}

template <typename T, int H, int RB, int NTZ, int MINB>
cudaError_t launch_zadj_v(const ZAdjArgs<T>& a, cudaStream_t st) {
  static PerDevice ready, cache;
  const size_t smem = sizeof(V2<T>) * (9 * RB * (skew_ld(H) + z_row_cap<H>()) + z_tw_slots<H>());
  constexpr auto kernel = k_zadj<T, H, RB, NTZ, MINB>;
  cudaError_t e = once_per_device(ready, [&] {
    cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return e;
  const int nb = resident_grid(kernel, NTZ, smem, (a.nrows + RB - 1) / RB, cache);
  return launch_pdl(kernel, nb, NTZ, smem, st, a);
}

template <int H, bool DA> cudaError_t launch_zadjw_v(const ZAdjArgs<float>& a, cudaStream_t st) {
  static PerDevice ready, cache;
  using Z = ZW<H>;
  auto smem_of = [](int Mzp) {
    return sizeof(float2) * (Z::TWS + (size_t)ZA_WARPS * (9 * Z::ROWS * Mzp + Z::ROWS * Z::XS));
  };
  const size_t smem = smem_of(a.Mzp), smax = smem_of(DA ? a.Mzp : H + 8);
  constexpr auto kernel = k_zadjw<H, DA>;
  cudaError_t e = once_per_device(ready, [&] {
    cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax);
    if (r != cudaSuccess) return r;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return e;
  const long long groups = a.nrows / Z::ROWS;
  const int nb = resident_grid(kernel, ZA_WARPS * 32, smax, (groups + ZA_WARPS - 1) / ZA_WARPS, cache);
  return launch_pdl(kernel, nb, ZA_WARPS * 32, smem, st, a);
}

template <int H> cudaError_t launch_zadjw(const ZAdjArgs<float>& a, cudaStream_t st) {
  const bool da = a.Mz == zw_da_mz<H>() && a.Mzp == (zw_da_mz<H>() + 7) / 8 * 8;
  return da ? launch_zadjw_v<H, true>(a, st) : launch_zadjw_v<H, false>(a, st);
}

// Rows per group of the generic form: nine fields of a group in about 60 KB.
template <typename T, int H> constexpr int zadj_rows() {
  constexpr int per = 9 * (skew_ld(H) + z_row_cap<H>()) * (int)sizeof(V2<T>);
  return per > 32768 ? 1 : (per > 16384 ? 2 : (per > 8192 ? 4 : 8));
}

template <typename T> cudaError_t launch_zadj(int H, const ZAdjArgs<T>& a, cudaStream_t st) {
  if constexpr (std::is_same<T, float>::value) {
    const int rows = H <= 256 ? 256 / H : 1;
    if (H >= 32 && H <= 256 && a.nrows % rows == 0 && a.Mzp % 8 == 0 && a.Mzp <= H + 8 && a.Mz <= a.Mzp) {
      if (H == 32) return launch_zadjw<32>(a, st);
      if (H == 64) return launch_zadjw<64>(a, st);
      if (H == 128) return launch_zadjw<128>(a, st);
      return launch_zadjw<256>(a, st);
    }
  }
  return dispatch_half(H, [&](auto hh) {
    constexpr int HH = decltype(hh)::value;
    constexpr int RB = zadj_rows<T, HH>();
    // about one last-stage butterfly of the forward transforms per thread
    constexpr int NBF = 6 * RB * (HH / fft16_radix(HH, fft16_nstages(HH) - 1));
    constexpr int NTZ = NBF <= 96 ? 96 : (NBF <= 192 ? 192 : 256);
    return launch_zadj_v<T, HH, RB, NTZ, 1>(a, st);
  });
}

template cudaError_t launch_zadj<float>(int, const ZAdjArgs<float>&, cudaStream_t);
template cudaError_t launch_zadj<double>(int, const ZAdjArgs<double>&, cudaStream_t);

}  // namespace hit
