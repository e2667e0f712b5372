// Warp-resident half-row transforms with 16 values per lane (float32, H =
// Nz/2 in {128, 256}): radix 16 over stride H/16, one exchange, then radix
// H/16 over stride 16.  LPR = H/16 lanes serve a row; lane b reads positions b +
// LPR r (r < 16) and ends with the same positions, so products of physical
// fields stay in the lane and are the next transform's inputs, as in zwarp.cuh
// -- whose three stages of 8 values per lane cross shared memory twice.
//
// Exchange slot p + p / 16, H + H/16 slots per row: the first stage's stores
// 16 b + r and the second stage's loads b + LPR h + 16 r of a half warp (16 /
// LPR rows) hit 16 distinct bank pairs.
#pragma once

#include "fft_core.cuh"

namespace hit {

template <int H> struct Z16 {
  static_assert(H == 128 || H == 256, "16-value rows");
  static constexpr int LPR = H / 16;          // lanes per row = radix of the second stage
  static constexpr int ROWS = 32 / LPR;       // rows per warp
  static constexpr int NBL = 16 / LPR;        // second-stage butterflies per lane
  static constexpr int XS = H + H / 16;       // exchange slots per row
  static constexpr int NTW = NBL * (LPR - 1); // second-stage twiddles of a lane
};

// Second-stage twiddles w_H^{r j}, j = b + LPR h, at [h (LPR - 1) + r - 1]:
// the same for every row and transform of the lane.
template <int H> __device__ __forceinline__ void z16_twiddles(float2 (&w)[Z16<H>::NTW], const float2* tw, int b) {
  using Z = Z16<H>;
#pragma unroll
  for (int h = 0; h < Z::NBL; ++h)
#pragma unroll
    for (int r = 1; r < Z::LPR; ++r) w[h * (Z::LPR - 1) + r - 1] = tw[r * (b + Z::LPR * h) * (TWN / H)];
}

template <int H, bool INV>
__device__ __forceinline__ void z16_transform(float2 (&v)[16], float2* xch, const float2 (&w)[Z16<H>::NTW], int b) {
  using Z = Z16<H>;
  DFT<16, INV, float2>::run(v);
#pragma unroll
  for (int r = 0; r < 16; ++r) xch[17 * b + r] = v[r];
  __syncwarp();
  float2 u[Z::NBL][Z::LPR];
#pragma unroll
  for (int h = 0; h < Z::NBL; ++h)
#pragma unroll
    for (int r = 0; r < Z::LPR; ++r) u[h][r] = xch[b + Z::LPR * h + 17 * r];
  __syncwarp();
#pragma unroll
  for (int h = 0; h < Z::NBL; ++h) {
#pragma unroll
    for (int r = 1; r < Z::LPR; ++r) {
      float2 t = w[h * (Z::LPR - 1) + r - 1];
      if (INV) t.y = -t.y;
      u[h][r] = cmul(u[h][r], t);
    }
    DFT<Z::LPR, INV, float2>::run(u[h]);
#pragma unroll
    for (int r = 0; r < Z::LPR; ++r) v[h + Z::NBL * r] = u[h][r];
  }
}

// e^{-2 pi i k / (2H)} at k = b + (H/16) r from w0 = e^{-2 pi i b / (2H)}: w0
// times e^{-i pi r / 16} (r a constant in unrolled loops).
__device__ __forceinline__ float2 z16_wz(float2 w0, int r) {
  constexpr float c[9] = {1.f, 0.98078528040323044913f, 0.92387953251128675613f, 0.83146961230254523708f,
                          0.70710678118654752440f, 0.55557023301960222474f, 0.38268343236508977173f,
                          0.19509032201612826785f, 0.f};
  if (r == 0) return w0;
  if (r == 8) return make_float2(w0.y, -w0.x);
  const float cr = r < 8 ? c[r] : -c[16 - r], ci = r < 8 ? -c[8 - r] : -c[r - 8];
  return cmul(w0, make_float2(cr, ci));
}

}  // namespace hit
