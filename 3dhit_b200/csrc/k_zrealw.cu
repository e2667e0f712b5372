// Warp-resident z passes of the 3-D transforms (float32 rows of 64 .. 512
// points): c2r and r2c of to_physical / to_spectral on the row transforms of
// zwarp.cuh.  A warp owns 256 / H rows; loads and stores are the lanes' own
// (256-byte runs), nothing is staged: at 60-odd registers the SM holds enough
// warps to cover the latency, and the conjugate partner's second read of a row
// hits L1.  The CTA-per-row-group kernels (k_zreal, k_zr2c) crossed shared
// memory under CTA barriers: three components of 256^3 took 111 (c2r) and 136
// us (r2c) for 404 MB, 0.56 and 0.45 of HBM.
#include "zrow.cuh"
#include "zwarp.cuh"

namespace hit {

constexpr int ZRW_WARPS = 4;

template <int H> struct ZrwRow {  // what a lane keeps for all rows
  using Z = ZW<H>;
  int q, b;
  float2* xch;
  float2 wl[7], wz0;
  ZwMid<H> mid;
  __device__ __forceinline__ ZrwRow(float2* tws, const float2* tw)
      : q((threadIdx.x & 31) / Z::LPR), b((threadIdx.x & 31) % Z::LPR), mid(b) {
    xch = tws + Z::TWS + ((threadIdx.x >> 5) * Z::ROWS + q) * Z::XS;
    zw_fill_twiddles<H, ZRW_WARPS * 32>(tws, tw);
    __syncthreads();
    zw_last_twiddles<H>(wl, tws, b);
    mid.load(tws);
    wz0 = tws[Z::TWZ + b];  // e^{-2 pi i k / Nz} of k = b + (H/8) r: zw_wz(wz0, r)
  }
};

template <int H>
__global__ void __launch_bounds__(ZRW_WARPS * 32, 6) k_zc2rw(ZRealArgs<float> a, long long ngroups, long long per_comp) {
  using Z = ZW<H>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tws = reinterpret_cast<float2*>(smem_raw);
  const ZrwRow<H> L(tws, a.tw);
  const int b = L.b, Mz = a.Mz;
  for (long long g = (long long)blockIdx.x * ZRW_WARPS + (threadIdx.x >> 5); g < ngroups;
       g += (long long)gridDim.x * ZRW_WARPS) {
    const long long c = g / per_comp, row = (g % per_comp) * Z::ROWS + L.q;
    const float2* in = a.cbuf + c * a.cc_stride + row * a.Mzp;
    float2 X[8], Y[8], v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int k = b + Z::NB0 * r, kk = H - k;
      X[r] = k < Mz ? __ldg(in + k) : make_float2(0.f, 0.f);
      Y[r] = kk < Mz ? __ldg(in + kk) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {  // see c2r_pre
      if (b + Z::NB0 * r == 0) {
        X[r].y = 0.f;
        Y[r].y = 0.f;
      }
      Y[r].y = -Y[r].y;
      float2 w = zw_wz(L.wz0, r);
      w.y = -w.y;
      v[r] = cadd(cadd(X[r], Y[r]), cmul_i(cmul(w, csub(X[r], Y[r]))));
    }
    zw_transform<H, true>(v, L.xch, tws, b, L.mid, L.wl);
    float2* out = reinterpret_cast<float2*>(a.rbuf + c * a.rc_stride + row * (2 * H));
#pragma unroll
    for (int r = 0; r < 8; ++r) out[b + Z::NB0 * r] = cscale(v[r], a.scale);
  }
}

template <int H>
__global__ void __launch_bounds__(ZRW_WARPS * 32, 6) k_zr2cw(ZRealArgs<float> a, long long ngroups, long long per_comp) {
  using Z = ZW<H>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tws = reinterpret_cast<float2*>(smem_raw);
  const ZrwRow<H> L(tws, a.tw);
  const int b = L.b, partner = L.q * Z::LPR + ((Z::LPR - b) & (Z::LPR - 1));
  const float2 wh = tws[Z::TWZ + H];
  for (long long g = (long long)blockIdx.x * ZRW_WARPS + (threadIdx.x >> 5); g < ngroups;
       g += (long long)gridDim.x * ZRW_WARPS) {
    const long long c = g / per_comp, row = (g % per_comp) * Z::ROWS + L.q;
    const float2* in = reinterpret_cast<const float2*>(a.rbuf + c * a.rc_stride + row * (2 * H));
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = __ldg(in + b + Z::NB0 * r);
    zw_transform<H, false>(v, L.xch, tws, b, L.mid, L.wl);
    float2* out = a.cbuf + c * a.cc_stride + row * a.Mzp;
#pragma unroll
    for (int r = 0; r < 8; ++r) {  // see r2c_post
      float2 t;
      t.x = __shfl_sync(0xffffffffu, v[7 - r].x, partner);
      t.y = __shfl_sync(0xffffffffu, v[7 - r].y, partner);
      float2 bc = b == 0 ? v[(8 - r) & 7] : t;
      bc.y = -bc.y;
      const float2 E = cscale(cadd(v[r], bc), 0.5f), O = cscale(cmul_mi(csub(v[r], bc)), 0.5f);
      out[b + Z::NB0 * r] = cadd(E, cmul(zw_wz(L.wz0, r), O));
    }
    for (int k = b; k < a.Mzp - H; k += Z::LPR) {  // bin H and the row's padding
      float2 x = make_float2(0.f, 0.f);
      if (k == 0) {
        float2 bc = v[0];
        bc.y = -bc.y;
        x = cadd(cscale(cadd(v[0], bc), 0.5f), cmul(wh, cscale(cmul_mi(csub(v[0], bc)), 0.5f)));
      }
      out[H + k] = x;
    }
  }
}

template <int H, bool C2R> cudaError_t launch_zrealw_v(const ZRealArgs<float>& a, int ncomp, cudaStream_t st) {
  using Z = ZW<H>;
  constexpr size_t smem = sizeof(float2) * (Z::TWS + (size_t)ZRW_WARPS * Z::ROWS * Z::XS);
  static PerDevice cache;
  const long long per = a.nrows / Z::ROWS, groups = per * ncomp, ctas = (groups + ZRW_WARPS - 1) / ZRW_WARPS;
  if constexpr (C2R) {
    const int grid = resident_grid(k_zc2rw<H>, ZRW_WARPS * 32, smem, ctas, cache);
    k_zc2rw<H><<<grid, ZRW_WARPS * 32, smem, st>>>(a, groups, per);
  } else {
    const int grid = resident_grid(k_zr2cw<H>, ZRW_WARPS * 32, smem, ctas, cache);
    k_zr2cw<H><<<grid, ZRW_WARPS * 32, smem, st>>>(a, groups, per);
  }
  return cudaGetLastError();
}

bool zrealw_ok(int H, const ZRealArgs<float>& a) {
  // whole row groups per warp, 8-byte aligned rows, padding of a full row (r2c writes it)
  return H >= 32 && H <= 256 && a.nrows % (256 / H) == 0 && a.Mz == H + 1 && a.Mzp >= H + 1 &&
         ((uintptr_t)a.cbuf % 8) == 0 && ((uintptr_t)a.rbuf % 8) == 0;
}
cudaError_t launch_zc2rw(int H, const ZRealArgs<float>& a, int ncomp, cudaStream_t st) {
  if (H == 32) return launch_zrealw_v<32, true>(a, ncomp, st);
  if (H == 64) return launch_zrealw_v<64, true>(a, ncomp, st);
  if (H == 128) return launch_zrealw_v<128, true>(a, ncomp, st);
  return launch_zrealw_v<256, true>(a, ncomp, st);
}
cudaError_t launch_zr2cw(int H, const ZRealArgs<float>& a, int ncomp, cudaStream_t st) {
  if (H == 32) return launch_zrealw_v<32, false>(a, ncomp, st);
  if (H == 64) return launch_zrealw_v<64, false>(a, ncomp, st);
  if (H == 128) return launch_zrealw_v<128, false>(a, ncomp, st);
  return launch_zrealw_v<256, false>(a, ncomp, st);
}

}  // namespace hit
