// Pointwise MLP of the learned subgrid-stress closure on the fifth-generation
// tensor cores: 9 -> 64 -> 64 -> 64 -> 6, GELU between layers, bf16 weights
// and activations, float32 accumulation in TMEM.
//
// Persistent CTAs of 128 threads work on 128-point tiles; thread t owns point
// t of the tile (its TMEM lane).  The weight operands stay in shared memory in
// the K-major core-matrix layout (tc_common.cuh).
//
// k_mlp (inference): one mlp::infer_tile per tile, 64 TMEM columns, as many
// CTAs per SM as shared memory and registers allow.
//
// k_mlp_train (training and vector-Jacobian products), per tile:
//   forward   z1 = [x, 0, 1] W1 (bias in row 15), a_l = gelu(z_l),
//             z_l = a_{l-1} W_l + b_l (l = 2, 3), y = a3 W4 + b4;
//   backward  dy = 2 (y - tau) / (P * 6) (the MSE loss) or the given cotangent,
//             da_{l-1} = dz_l W_l^T, dz_{l-1} = da_{l-1} * gelu'(z_{l-1});
//   weights   dW_l += a_{l-1}^T dz_l in TMEM accumulators that live as long as
//             the CTA (its partial sums go out once, at the end).
// The activation tiles [point][feature] serve twice: K-major for the layers,
// and, read with the points as the contracted dimension, as the MN-major
// operands of the weight gradients (tc::smem_desc with the two strides
// swapped), so neither activations nor gradients leave the SM.  Before, they
// were written feature-major (419 rows of 2-byte stores per point) and read
// back by four GEMMs: 4.19 M points took 3.0 ms in the pass and 4.9 ms in the
// GEMMs, with 3.5 GB of workspace each way.  The whole gradient now takes 1.69
// ms (133 TFLOP/s); what bounds it is the chain of ten MMA round trips per tile
// at two CTAs per SM, and the 384 hardware tanh per point.
// TMEM (256 columns, so that two CTAs share an SM): [0, 64) layer
// accumulators; dW2, dW3 64 columns each; then 16 each for dz1^T x, dz2^T x,
// dz3^T x (column 15 of x is 1: the bias gradients; all of dW1 for dz1) and
// a3^T dz4.  No room is left to keep z1..z3, so the backward forms z_l again
// beside da_l (the same operands, the same sums), 32 columns of each at a time.
// An accumulator of 64 rows is computed as one of 128: its A operand runs on
// into whatever lies behind the tile, and lanes 64..127 are not read.
// Shared memory: dz3, dz2, dz1 overwrite a3, a2, a1 once the MMAs that read
// those are complete.
#include <cuda_bf16.h>

#include <algorithm>

#include "kernels.h"
#include "mlp_core.cuh"
#include "tc_common.cuh"

namespace hit {

using namespace mlp;

namespace {
constexpr int MLP_WAIT = 1 << 22;
}  // namespace

__global__ void __launch_bounds__(128) k_mlp(MlpArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  InferSmem& S = *reinterpret_cast<InferSmem*>(smem_raw);
  infer_setup(S, a.w1t, a.w2t, a.w3t, a.w4t, a.b2, a.b3, a.b4);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  uint32_t phase = 0;
  bool ok = true;
  for (long long tile = blockIdx.x; tile * 128 < a.P && ok; tile += gridDim.x) {
    const long long p = tile * 128 + threadIdx.x;
    const bool in = p < a.P;
    float x[9], y[6];
#pragma unroll
    for (int i = 0; i < 9; ++i) x[i] = in ? a.x[i * a.x_sf + p * a.x_sp] : 0.f;
    infer_tile(S, x, y, phase, ok, MLP_WAIT);
    if (in) {
#pragma unroll
      for (int i = 0; i < 6; ++i) a.y[i * a.y_sf + p * a.y_sp] = y[i];
    }
  }
  if (!ok && threadIdx.x == 0) atomicExch(a.err, 1);
  infer_teardown(S);
}

struct TrainSmem {
  unsigned char w1t[64 * 16 * 2], w2t[64 * 64 * 2], w3t[64 * 64 * 2], w4t[16 * 64 * 2];
  unsigned char w4[64 * 16 * 2], w3[64 * 64 * 2], w2[64 * 64 * 2];  // backward operands
  unsigned char w1[16 * 64 * 2];  // backward layer 1 (input gradient, vector-Jacobian mode)
  unsigned char a1[128 * 64 * 2], a2[128 * 64 * 2], a3[128 * 64 * 2];
  unsigned char x0[2][128 * 16 * 2];  // layer input (the last tile's is read by its dW1 after the next has begun)
  unsigned char dz4[128 * 16 * 2];
  float b2[64], b3[64], b4[16];
  double red[4];
  uint64_t mbar;
  uint32_t tslot;
};

// columns [c, c + 8) of row `row` of a K-major tile with 64 columns
__device__ __forceinline__ void store_bf16x8(unsigned char* tile, int row, int c, const float* v) {
  uint4 q;
  uint32_t* w = reinterpret_cast<uint32_t*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(tile + tc::kmajor_off(row, c, 64)) = q;
}

__global__ void __launch_bounds__(128, 2) k_mlp_train(MlpArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
  constexpr uint32_t DW2 = 64, DW3 = 128, S1 = 192, S2 = 208, S3 = 224, S4 = 240, NCOL = 256;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t mb = tc::smem_u32(&S.mbar);
  // weights and biases (resident for all tiles)
  load_kmajor(S.w1t, a.w1t, 64, 16);
  load_kmajor(S.w2t, a.w2t, 64, 64);
  load_kmajor(S.w3t, a.w3t, 64, 64);
  load_kmajor(S.w4t, a.w4t, 16, 64);
  load_kmajor(S.w4, a.w4, 64, 16);
  load_kmajor(S.w3, a.w3, 64, 64);
  load_kmajor(S.w2, a.w2, 64, 64);
  if (a.xbar) load_kmajor(S.w1, a.w1, 16, 64);
  for (int i = tid; i < 64; i += 128) {
    S.b2[i] = a.b2[i];
    S.b3[i] = a.b3[i];
  }
  if (tid < 16) S.b4[tid] = a.b4[tid];
  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&S.tslot), NCOL);
  if (tid == 0) tc::mbar_init(mb, 1);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = S.tslot;
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's TMEM lanes
  uint32_t phase = 0;
  bool ok = true;
  double loss = 0.0, db4[6] = {0, 0, 0, 0, 0, 0};
  const uint32_t id64 = tc::idesc_bf16(128, 64), id32 = tc::idesc_bf16(128, 32), id16 = tc::idesc_bf16(128, 16);
  const uint32_t it64 = tc::idesc_bf16_tt(128, 64), it16 = tc::idesc_bf16_tt(128, 16);

  // Thread 0 issues the MMAs of `issue` once every thread's shared-memory
  // writes are visible, and every thread waits for their completion (bounded;
  // after a wait gave up, nothing more is issued).
  auto round = [&](auto&& issue) {
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && ok) {
      issue();
      tc::commit(mb);
    }
    ok = __syncthreads_and(ok && tc::mbar_wait(mb, phase, MLP_WAIT)) != 0;  // block-uniform
    phase ^= 1;
    tc::fence_after_sync();
  };
  // D[col..] = A B^T: A a K-major tile of KA columns, B K-major rows of KB columns
  auto layer = [&](uint32_t col, const unsigned char* A, int KA, const unsigned char* B, int KB, int steps,
                   uint32_t idesc) {
    const uint32_t a0 = tc::smem_u32(A), b0 = tc::smem_u32(B);
    for (int s = 0; s < steps; ++s)
      tc::mma_bf16(tmem + col, tc::smem_desc(a0 + 256 * s, 128, KA * 16), tc::smem_desc(b0 + 256 * s, 128, KB * 16),
                   idesc, s > 0);
  };
  // D[col..] (+)= A^T B over the tile's 128 points: both operands are
  // [point][feature] tiles read MN-major (8-feature groups 128 bytes apart,
  // 8-point groups K * 16 bytes apart, two of those per MMA)
  bool first = true;  // no tile accumulated yet
  auto grad = [&](uint32_t col, const unsigned char* A, const unsigned char* B, int KB, uint32_t idesc, bool acc) {
    const uint32_t a0 = tc::smem_u32(A), b0 = tc::smem_u32(B);
    for (int s = 0; s < 8; ++s)
      tc::mma_bf16(tmem + col, tc::smem_desc(a0 + 2048 * s, 1024, 128),
                   tc::smem_desc(b0 + 2 * KB * 16 * s, KB * 16, 128), idesc, acc || s > 0);
  };
  // a_l = gelu(z_l + bias) from the accumulator into its tile, 16 columns at a time
  auto act = [&](unsigned char* dst, const float* bias) {
#pragma unroll
    for (int c = 0; c < 64; c += 16) {
      float t[16];
      tc::tmem_ld16(lane_base + c, t);
#pragma unroll
      for (int i = 0; i < 16; ++i) t[i] = gelu(t[i] + (bias ? bias[c + i] : 0.f));
      store_bf16x8(dst, tid, c, t);
      store_bf16x8(dst, tid, c + 8, t + 8);
    }
  };
  // columns [32 h, 32 h + 32) of dz_l from da (TMEM columns 0..31) and z (32..63)
  auto back = [&](unsigned char* dst, int h, const float* bias) {
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      float d[16], z[16];
      tc::tmem_ld16(lane_base + c, d);
      tc::tmem_ld16(lane_base + 32 + c, z);
#pragma unroll
      for (int i = 0; i < 16; ++i) d[i] *= gelu_d(z[i] + (bias ? bias[32 * h + c + i] : 0.f));
      store_bf16x8(dst, tid, 32 * h + c, d);
      store_bf16x8(dst, tid, 32 * h + c + 8, d + 8);
    }
  };
  // da_l and z_l, columns [32 h, 32 h + 32): B rows 32 h .. (four 8-row groups on)
  auto back_mma = [&](const unsigned char* dz, int KD, const unsigned char* w, const unsigned char* prev, int KP,
                      const unsigned char* wt, int h) {
    layer(0, dz, KD, w + 4 * h * KD * 16, KD, KD / 16, id32);
    layer(32, prev, KP, wt + 4 * h * KP * 16, KP, KP / 16, id32);
  };

  int xb = 0;            // x0 buffer of the current tile
  bool pending = false;  // the last tile's dW1 is still to be issued
  for (long long tile = blockIdx.x; tile * 128 < a.P && ok; tile += gridDim.x) {
    const long long p = tile * 128 + tid;
    const bool in = p < a.P;
    unsigned char* x0 = S.x0[xb];
    {
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = 0.f;
      if (in) {
#pragma unroll
        for (int i = 0; i < 9; ++i) x[i] = a.x[i * a.x_sf + p * a.x_sp];
      }
      x[15] = in ? 1.f : 0.f;  // bias input of layer 1
      store_row<16>(x0, tid, x, 16);
    }
    // ---- forward ----
    round([&] {
      if (pending) grad(S1, S.a1, S.x0[xb ^ 1], 16, it16, !first);  // last tile: dz1 (in a1), x
      layer(0, x0, 16, S.w1t, 16, 1, id64);
    });
    if (pending) first = false;
    act(S.a1, nullptr);
    round([&] { layer(0, S.a1, 64, S.w2t, 64, 4, id64); });
    act(S.a2, S.b2);
    round([&] { layer(0, S.a2, 64, S.w3t, 64, 4, id64); });
    act(S.a3, S.b3);
    round([&] { layer(0, S.a3, 64, S.w4t, 64, 4, id16); });
    {
      float y[16], dz[16];
      tc::tmem_ld16(lane_base, y);
#pragma unroll
      for (int i = 0; i < 16; ++i) dz[i] = 0.f;
#pragma unroll
      for (int i = 0; i < 6; ++i) y[i] += S.b4[i];
      if (in && a.ybar) {  // vector-Jacobian mode: the upstream dL/dy
#pragma unroll
        for (int i = 0; i < 6; ++i) dz[i] = a.ybar[i * a.yb_sf + p * a.yb_sp];
      } else if (in) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const float r = y[i] - a.tau[p * 6 + i];
          loss += (double)r * r;
          dz[i] = 2.f * r * a.inv_count;
        }
      }
      // (of the bf16 values that the weight gradients contract, as for the other biases)
#pragma unroll
      for (int i = 0; i < 6; ++i) db4[i] += (double)__bfloat162float(__float2bfloat16_rn(dz[i]));
      store_row<16>(S.dz4, tid, dz, 16);
    }
    // ---- backward, two halves of 32 columns per layer ----
    const bool acc = pending;  // an earlier tile has been accumulated
    round([&] {
      grad(S4, S.a3, S.dz4, 16, it16, acc);
      back_mma(S.dz4, 16, S.w4, S.a2, 64, S.w3t, 0);
    });
    back(S.a3, 0, S.b3);
    round([&] { back_mma(S.dz4, 16, S.w4, S.a2, 64, S.w3t, 1); });
    back(S.a3, 1, S.b3);  // a3 holds dz3
    round([&] {
      grad(DW3, S.a2, S.a3, 64, it64, acc);
      grad(S3, S.a3, x0, 16, it16, acc);
      back_mma(S.a3, 64, S.w3, S.a1, 64, S.w2t, 0);
    });
    back(S.a2, 0, S.b2);
    round([&] { back_mma(S.a3, 64, S.w3, S.a1, 64, S.w2t, 1); });
    back(S.a2, 1, S.b2);  // a2 holds dz2
    round([&] {
      grad(DW2, S.a1, S.a2, 64, it64, acc);
      grad(S2, S.a2, x0, 16, it16, acc);
      back_mma(S.a2, 64, S.w2, x0, 16, S.w1t, 0);
    });
    back(S.a1, 0, nullptr);
    round([&] { back_mma(S.a2, 64, S.w2, x0, 16, S.w1t, 1); });
    back(S.a1, 1, nullptr);  // a1 holds dz1
    if (a.xbar) {  // dx = dz1 W1
      round([&] { layer(0, S.a1, 64, S.w1, 64, 4, id16); });
      float dx[16];
      tc::tmem_ld16(lane_base, dx);
      if (in) {
#pragma unroll
        for (int i = 0; i < 9; ++i) a.xbar[i * a.x_sf + p * a.x_sp] = dx[i];
      }
    }
    pending = true;
    xb ^= 1;
  }
  if (pending) round([&] { grad(S1, S.a1, S.x0[xb ^ 1], 16, it16, !first); });
  if (!ok && tid == 0) atomicExch(a.err, 1);

  // partial sums of this CTA: dW1 [16][64], dW2, dW3 [65][64], dW4 [65][16]
  // (lane i of an accumulator is row i)
  float* part = a.part + (long long)blockIdx.x * MLP_PART;
  if (warp < 2) {
    const int i = tid;
#pragma unroll 1
    for (int l = 0; l < 2; ++l) {
      float* dw = part + 1024 + l * 65 * 64;
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        float t[16];
        tc::tmem_ld16(lane_base + (l ? DW3 : DW2) + c, t);
#pragma unroll
        for (int k = 0; k < 16; ++k) dw[i * 64 + c + k] = t[k];
      }
      float t[16];
      tc::tmem_ld16(lane_base + (l ? S3 : S2), t);
      dw[64 * 64 + i] = t[15];
    }
    float t[16];
    tc::tmem_ld16(lane_base + S1, t);
#pragma unroll
    for (int k = 0; k < 16; ++k) part[k * 64 + i] = t[k];
    tc::tmem_ld16(lane_base + S4, t);
    float* dw4 = part + 1024 + 2 * 65 * 64;
#pragma unroll
    for (int k = 0; k < 16; ++k) dw4[i * 16 + k] = t[k];
    if (tid < 10) dw4[64 * 16 + 6 + tid] = 0.f;
  }
  // the loss and db4: warp sums, then the four warps in order
  auto cta_sum = [&](double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) S.red[warp] = v;
    __syncthreads();
    return S.red[0] + S.red[1] + S.red[2] + S.red[3];
  };
  for (int i = 0; i < 6; ++i) {
    const double v = cta_sum(db4[i]);
    if (tid == 0) part[1024 + 2 * 65 * 64 + 64 * 16 + i] = (float)v;
  }
  const double v = cta_sum(loss);
  if (tid == 0 && a.loss) a.loss[blockIdx.x] = v;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, NCOL);
}

// Sums of the CTAs' partials, one warp per 32 consecutive values (coalesced),
// 8 warps sharing the partials, added in warp order in float64; the loss by
// the last block.
constexpr int MS_W = 8;
__global__ void __launch_bounds__(MS_W * 32) k_mlp_sums(MlpSumArgs a) {
  __shared__ double red[MS_W][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + lane;
  const bool is_loss = blockIdx.x == gridDim.x - 1;
  double s = 0.0;
  if (is_loss) {
    if (a.loss)
      for (int b = warp * 32 + lane; b < a.nparts; b += MS_W * 32) s += a.loss_part[b];
  } else if (v < MLP_PART) {
#pragma unroll 8
    for (int b = warp; b < a.nparts; b += MS_W) s += (double)a.part[(long long)b * MLP_PART + v];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
    s = 0.0;
#pragma unroll
    for (int w = 0; w < MS_W; ++w) s += red[w][lane];
    if (is_loss) {
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0 && a.loss) *a.loss = s * a.loss_scale;
    } else if (v < MLP_PART) {
      const float f = (float)s;
      if (v < 1024) a.dW1[v] = f;
      else if (v < 1024 + 65 * 64) a.dW2[v - 1024] = f;
      else if (v < 1024 + 2 * 65 * 64) a.dW3[v - 1024 - 65 * 64] = f;
      else a.dW4[v - 1024 - 2 * 65 * 64] = f;
    }
  }
}

cudaError_t launch_mlp_train(const MlpArgs& a, int grid, cudaStream_t st) {
  static PerDevice ready;
  cudaError_t e = once_per_device(ready, [] {
    cudaError_t r = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(TrainSmem));
    if (r != cudaSuccess) return r;
    return cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return e;
  k_mlp_train<<<grid, 128, sizeof(TrainSmem), st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mlp_sums(const MlpSumArgs& a, cudaStream_t st) {
  k_mlp_sums<<<(MLP_PART + 31) / 32 + 1, MS_W * 32, 0, st>>>(a);
  return cudaGetLastError();
}

// Inference.  grid = 0: one resident wave of CTAs (at most 8 per SM: 8 x 64
// TMEM columns fill the SM's 512), or -k: k CTAs per SM (a lighter footprint
// next to other work on the GPU).
cudaError_t launch_mlp(const MlpArgs& a, int grid, cudaStream_t st) {
  // per device: the attribute set-up and the wave (CTAs per SM, and that times
  // the SM count)
  static PerDevice ready, wave_of, per_sm_of;
  const int smem = (int)sizeof(InferSmem);
  cudaError_t e = once_per_device(ready, [&] {
    // the largest shared-memory carveout, so that the occupancy below (and the
    // launch) can place several CTAs per SM
    cudaError_t r = cudaFuncSetAttribute(k_mlp, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (r != cudaSuccess) return r;
    return cudaFuncSetAttribute(k_mlp, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return e;
  std::atomic<int>* ws = wave_of.here();
  std::atomic<int>* ps = per_sm_of.here();
  int wave = ws ? ws->load(std::memory_order_relaxed) : 0;
  int per_sm_wave = ps ? ps->load(std::memory_order_relaxed) : 0;
  if (wave == 0 || per_sm_wave == 0) {
    // CTAs per SM from the SM's shared memory and registers (1 KB of
    // shared memory per CTA is the driver's)
    int dev = 0, sms = 0, smem_sm = 0, regs_sm = 0;
    cudaFuncAttributes fa{};
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess)
      return e;
    if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncGetAttributes(&fa, k_mlp)) != cudaSuccess) return e;
    const int by_smem = smem_sm / (smem + 1024);
    const int by_regs = regs_sm / (128 * ((std::max(fa.numRegs, 1) + 7) / 8 * 8));
    per_sm_wave = std::max(1, std::min(std::min(by_smem, by_regs), 8));
    wave = per_sm_wave * sms;
    if (ps) ps->store(per_sm_wave, std::memory_order_relaxed);
    if (ws) ws->store(wave, std::memory_order_relaxed);
  }
  const long long tiles = (a.P + 127) / 128;
  if (grid < 0) grid = (int)std::min<long long>(tiles, std::min(-grid * (wave / per_sm_wave), wave));
  if (grid <= 0) grid = (int)std::min<long long>(tiles, wave);
  k_mlp<<<grid, 128, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace hit
