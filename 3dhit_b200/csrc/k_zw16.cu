// k_zw16: the fused z pass of the RHS (as k_zwarp: c2r of u and w, u x w, r2c of
// the products, per (x, y) row) for the dealiased layout with 16 values per
// lane (zw16.cuh): each transform crosses shared memory once instead of twice.
// k_zwarp is bound by that data path (73 to 83% of its wavefronts in ncu).
// The three u fields of a row, 96 registers per lane, are parked in the lane's
// tensor memory (tcgen05.st / tcgen05.ld) between their uses; the products
// accumulate in registers (254 registers, two CTAs per SM).
// Z pass per launch: 512^3 1137 -> 928 us (0.53 of HBM), 256^3 143 -> 123, 128 x
// 64 x 256 26.9 -> 24.9.  Parking a product too and staging three fields at a
// time, for three CTAs per SM, measured slower (1047 us at 512^3: the tensor
// memory round trips and the extra staging waits).
#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "tc_common.cuh"
#include "tma.cuh"
#include "zrow.cuh"
#include "zw16.cuh"

namespace hit {

__device__ int g_zw16_timeout = 0;  // set when a TMA wait gave up (hit_device_status)
__device__ int g_zw16_wait_limit = Z_WAIT;  // polls of the wait for a row group (hit_set_wait_limit)

cudaError_t set_zw16_wait_limit(int polls) {
  const int v = polls < 0 ? Z_WAIT : polls;
  return cudaMemcpyToSymbol(g_zw16_wait_limit, &v, sizeof(int));
}
cudaError_t take_zw16_timeout(int* flag) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_zw16_timeout, sizeof(int));
  if (e != cudaSuccess) return e;
  *flag = v;
  const int zero = 0;
  return v ? cudaMemcpyToSymbol(g_zw16_timeout, &zero, sizeof(int)) : cudaSuccess;
}

constexpr int ZW16_WARPS = 4;
constexpr int ZW16_COLS = 128;  // TMEM columns per CTA (96 used: u0, u1, u2)

template <int H> struct Z16Row {
  static constexpr int MZ = zw_da_mz<H>(), MZP = (MZ + 7) / 8 * 8;
  static constexpr int SP = MZP;  // staged row pitch: the rows of a half warp start LPR bank pairs apart
  static_assert(H == 256 || SP % 16 == Z16<H>::LPR, "conflict-free rows");
  static constexpr int STG = 6 * Z16<H>::ROWS * SP;       // staged entries per warp
  static constexpr int XCH = Z16<H>::ROWS * Z16<H>::XS;   // exchange slots per warp
};

template <int H>
__global__ void __launch_bounds__(ZW16_WARPS * 32, 2) k_zw16(ZCrossArgs<float> a) {
  using Z = Z16<H>;
  using R = Z16Row<H>;
  constexpr int MZ = R::MZ, MZP = R::MZP, LPR = Z::LPR;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[ZW16_WARPS];
  __shared__ uint32_t tslot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = lane / LPR, b = lane % LPR;
  float2* stg = reinterpret_cast<float2*>(smem_raw) + warp * (R::STG + R::XCH);
  float2* xch = stg + R::STG + q * Z::XS;
  float2 w[Z::NTW];
  z16_twiddles<H>(w, a.tw, b);
  const float2 wz0 = a.tw[b * (TWN / (2 * H))];  // e^{-2 pi i b / Nz}
  const uint32_t mb = tma::smem_u32(&bars[warp]);
  if (lane == 0) tma::mbar_init(mb, 1);
  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tslot), ZW16_COLS);
  tma::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tm = tslot + ((uint32_t)(32 * warp) << 16);

  const int wait_limit = g_zw16_wait_limit;
  const long long ngroups = a.nrows / Z::ROWS;
  const long long nwarps = (long long)gridDim.x * ZW16_WARPS;
  constexpr uint32_t row_bytes = MZP * (uint32_t)sizeof(float2);
  auto prefetch = [&](long long grp) {
    if (lane == 0) tma::mbar_expect_tx(mb, 6u * Z::ROWS * row_bytes);
    __syncwarp();
    for (int i = lane; i < 6 * Z::ROWS; i += 32) {
      const int c = i / Z::ROWS, rr = i % Z::ROWS;
      tma::load_bytes(stg + i * R::SP, a.buf + c * a.c_stride + (grp * Z::ROWS + rr) * MZP, row_bytes, mb);
    }
  };
  pdl_wait();
  pdl_trigger();
  long long grp = (long long)blockIdx.x * ZW16_WARPS + warp;
  if (grp < ngroups) prefetch(grp);
  uint32_t phase = 0;
  const float s2 = 0.5f * a.scale * a.scale;  // both inverse normalisations and the r2c 1/2
  for (; grp < ngroups; grp += nwarps) {
    {
      const bool ok = __all_sync(0xffffffffu, tma::mbar_wait(mb, phase, wait_limit));
      phase ^= 1;
      if (!ok) {
        if (lane == 0) atomicExch(&g_zw16_timeout, 1);
        tma::mbar_wait(mb, phase ^ 1, Z_WAIT);  // the copies in flight, once more with a limit
        break;
      }
    }
    auto inverse = [&](int c, float2 (&v)[16]) {  // c2r of staged field c (see c2r_pre)
      const float2* row = stg + (c * Z::ROWS + q) * R::SP;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int k = b + LPR * r, kk = H - k, lo = LPR * r, hi = lo + LPR - 1;
        float2 X = hi < MZ || (lo < MZ && k < MZ) ? row[k] : make_float2(0.f, 0.f);
        float2 Y = H - lo < MZ || (H - hi < MZ && kk < MZ) ? row[kk] : make_float2(0.f, 0.f);
        if (k == 0) X.y = 0.f;
        Y.y = -Y.y;
        const float2 sm = cadd(X, Y), df = csub(X, Y);
        float2 t = z16_wz(wz0, r);
        t.y = -t.y;
        v[r] = cadd(sm, cmul_i(cmul(t, df)));
      }
      z16_transform<H, true>(v, xch, w, b);
    };
    auto park = [&](int f, const float2 (&v)[16]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float t[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          t[2 * i] = v[8 * h + i].x;
          t[2 * i + 1] = v[8 * h + i].y;
        }
        tc::tmem_st16(tm + 32 * f + 16 * h, t);
      }
    };
    // f(r, u_f[r]) over the parked field f
    auto parked = [&](int f, auto&& fn) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float t[16];
        tc::tmem_ld16(tm + 32 * f + 16 * h, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) fn(8 * h + i, make_float2(t[2 * i], t[2 * i + 1]));
      }
    };
    float2 v[16], n0[16], n1[16], n2[16];
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      inverse(c, v);
      park(c, v);
    }
    tc::tmem_wait_st();
    // u x w (navierstokes.py:82-86): n0 = u1 w2 - u2 w1, n1 = u2 w0 - u0 w2, n2 = u0 w1 - u1 w0
    inverse(3, v);
    parked(2, [&](int r, float2 u) { n1[r] = __fmul2_rn(u, v[r]); });
    parked(1, [&](int r, float2 u) { n2[r] = __fmul2_rn(u, make_float2(-v[r].x, -v[r].y)); });
    inverse(4, v);
    parked(2, [&](int r, float2 u) { n0[r] = __fmul2_rn(u, make_float2(-v[r].x, -v[r].y)); });
    parked(0, [&](int r, float2 u) {
      n2[r] = __fmul2_rn(__ffma2_rn(u, v[r], n2[r]), make_float2(s2, s2));
    });
    inverse(5, v);
    if (grp + nwarps < ngroups) prefetch(grp + nwarps);  // every lane is past its staged reads
    parked(1, [&](int r, float2 u) {
      n0[r] = __fmul2_rn(__ffma2_rn(u, v[r], n0[r]), make_float2(s2, s2));
    });
    parked(0, [&](int r, float2 u) {
      n1[r] = __fmul2_rn(__ffma2_rn(u, make_float2(-v[r].x, -v[r].y), n1[r]), make_float2(s2, s2));
    });
    // r2c of the three products, over the first three input fields
    const int partner = q * LPR + ((LPR - b) & (LPR - 1));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = c == 0 ? n0[r] : (c == 1 ? n1[r] : n2[r]);
      z16_transform<H, false>(v, xch, w, b);
      float2* out = a.buf + c * a.c_stride + (grp * Z::ROWS + q) * MZP;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int k = b + LPR * r, lo = LPR * r, hi = lo + LPR - 1;
        if (lo >= MZP) break;  // the bins past the row are not formed
        // Z[H - k]: lane (LPR - b) mod LPR of the row, value 15 - r; for b = 0
        // this lane's own value (16 - r) mod 16 (Z[H] = Z[0])
        float2 t;
        t.x = __shfl_sync(0xffffffffu, v[15 - r].x, partner);
        t.y = __shfl_sync(0xffffffffu, v[15 - r].y, partner);
        float2 bc = b == 0 ? v[(16 - r) & 15] : t;
        bc.y = -bc.y;
        const float2 E = cadd(v[r], bc), O = cmul_mi(csub(v[r], bc));
        float2 x = cadd(E, cmul(z16_wz(wz0, r), O));
        if (!(hi < MZ || k < MZ)) x = make_float2(0.f, 0.f);
        if (hi < MZP || k < MZP) out[k] = x;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tslot, ZW16_COLS);
}

template <int H> cudaError_t launch_zw16_v(const ZCrossArgs<float>& a, cudaStream_t st) {
  static PerDevice ready, cache;
  using R = Z16Row<H>;
  constexpr size_t smem = sizeof(float2) * (size_t)ZW16_WARPS * (R::STG + R::XCH) + 128;
  cudaError_t e = once_per_device(ready, [] {
    cudaError_t r = cudaFuncSetAttribute(k_zw16<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
    return cudaFuncSetAttribute(k_zw16<H>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return e;
  // resident CTAs from the SM's shared memory and registers (the occupancy
  // query counts one per SM for kernels that allocate tensor memory)
  std::atomic<int>* slot = cache.here();
  int wave = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (wave == 0) {
    int dev = 0, sms = 0, smem_sm = 0, regs_sm = 0;
    cudaFuncAttributes fa{};
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncGetAttributes(&fa, k_zw16<H>)) != cudaSuccess) return e;
    const int by_smem = smem_sm / (int)(smem + fa.sharedSizeBytes + 1024);
    const int by_regs = regs_sm / (ZW16_WARPS * 32 * ((std::max(fa.numRegs, 1) + 7) / 8 * 8));
    wave = std::max(1, std::min(std::min(by_smem, by_regs), 512 / ZW16_COLS)) * std::max(sms, 1);
    if (slot) slot->store(wave, std::memory_order_relaxed);
  }
  const long long ctas = (a.nrows / Z16<H>::ROWS + ZW16_WARPS - 1) / ZW16_WARPS;
  return launch_pdl(k_zw16<H>, (int)std::max(1LL, std::min<long long>(ctas, wave)), ZW16_WARPS * 32, smem, st, a);
}

// Rows of 256 and 512 points on the dealiased layout (rows of 128 points, eight
// to a warp, are faster on k_zwarp: 22.7 against 25.0 us at 128^3).
bool zw16_ok(int H, const ZCrossArgs<float>& a) {
  if (H != 128 && H != 256) return false;
  const int mz = 2 * H / 3 + 1;
  return a.Mz == mz && a.Mzp == (mz + 7) / 8 * 8 && a.nrows % (512 / H) == 0;
}
cudaError_t launch_zw16(int H, const ZCrossArgs<float>& a, cudaStream_t st) {
  if (H == 128) return launch_zw16_v<128>(a, st);
  return launch_zw16_v<256>(a, st);
}

}  // namespace hit
