// Layout conversion, elementwise spectral operators and the float64
// reductions (spectra, budget, forcing coefficients).
//
// Reductions are two-level and deterministic: each block writes its partial
// sums to a fixed slot, then one finaliser sums the slots in a fixed order
// with Kahan compensation.  Shell indices reproduce the reference's float
// arithmetic exactly: floor(sqrt(k2)/k0 + 0.5) with every operation rounded
// in the run dtype (src/hit3d/diagnostics.py:76-82).
#include "kernels.h"

namespace hit {

template <typename T> __device__ __forceinline__ int shell_of(T k2, T k0);
template <> __device__ __forceinline__ int shell_of<float>(float k2, float k0) {
  return (int)floorf(__fadd_rn(__fdiv_rn(__fsqrt_rn(k2), k0), 0.5f));
}
template <> __device__ __forceinline__ int shell_of<double>(double k2, double k0) {
  return (int)floor(__dadd_rn(__ddiv_rn(__dsqrt_rn(k2), k0), 0.5));
}

// Layout copies and the box check take a mode per thread, or, where it is faster
// (gather_by_rows, check_by_rows), whole (x, y) rows per warp, lanes along z,
// LC_UNROLL 32-mode chunks of the three components in flight per lane.  The
// row's coordinates and offsets are then formed once instead of with a division by
// each extent per mode, whose arithmetic bounds large float32 grids; rows shorter
// than a warp and grids with few rows leave lanes or warps idle.
constexpr int LC_UNROLL = 2;
constexpr int LC_WARPS = NT / 32;

// ---------------------------------------------------------------------------
// gather: reference layout -> compact layout (+ optional NSCAL partial sums)
// ---------------------------------------------------------------------------
template <typename T> struct GatherSums {  // a thread's share of the NSCAL sums
  double E = 0, O = 0, B = 0;
  __device__ __forceinline__ void add(const GatherArgs<T>& a, const V2<T> (&v)[3], T kx, T ky, int k) {
    const T k2 = k2_of(kx, ky, a.k.kz[k]);
    double a2 = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) a2 += (double)v[c].x * v[c].x + (double)v[c].y * v[c].y;
    const double w = herm_weight(a.g, k);
    E += w * a2;
    O += w * (double)k2 * a2;
    if (a.kmin2 <= k2 && k2 <= a.kmax2) B += w * a2;
  }
  __device__ __forceinline__ void store(const GatherArgs<T>& a, double* red) {
    double r = block_sum_f64(E, red);
    if (threadIdx.x == 0) a.partial[3 * blockIdx.x + 0] = r;
    r = block_sum_f64(O, red);
    if (threadIdx.x == 0) a.partial[3 * blockIdx.x + 1] = r;
    r = block_sum_f64(B, red);
    if (threadIdx.x == 0) a.partial[3 * blockIdx.x + 2] = r;
  }
};

template <typename T>
__global__ void __launch_bounds__(NT) k_gather(GatherArgs<T> a) {
  __shared__ double red[32];
  const Geom& g = a.g;
  const long long nmodes = (long long)g.Mx * g.My * g.Mzp;
  const long long ce = (long long)g.Nx * g.Ny * g.Nzh;  // ext comp stride
  const long long cc = (long long)g.Mx * g.My * g.Mzp;  // compact comp stride
  GatherSums<T> s;
  for (long long m = blockIdx.x * (long long)NT + threadIdx.x; m < nmodes; m += (long long)gridDim.x * NT) {
    const int k = (int)(m % g.Mzp);
    const long long r = m / g.Mzp;
    const int j = (int)(r % g.My), i = (int)(r / g.My);
    V2<T> v[3] = {czero<T>(), czero<T>(), czero<T>()};
    if (k < g.Mz) {
      const int fx = full_pos(i, g.hx, g.Mx, g.Nx), fy = full_pos(j, g.hy, g.My, g.Ny);
      const long long e = ((long long)fx * g.Ny + fy) * g.Nzh + k;
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = a.ext[c * ce + e];
      if (a.partial) s.add(a, v, a.k.kx[fx], a.k.ky[fy], k);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) a.cmp[c * cc + m] = v[c];
  }
  if (a.partial) s.store(a, red);
}

__global__ void __launch_bounds__(NT) k_gather_rows(GatherArgs<float> a) {
  __shared__ double red[32];
  const Geom& g = a.g;
  const long long ce = (long long)g.Nx * g.Ny * g.Nzh;  // ext comp stride
  const long long cc = (long long)g.Mx * g.My * g.Mzp;  // compact comp stride
  const int lane = threadIdx.x & 31, nrows = g.Mx * g.My;
  GatherSums<float> s;
  for (int row = blockIdx.x * LC_WARPS + (threadIdx.x >> 5); row < nrows; row += gridDim.x * LC_WARPS) {
    const int j = row % g.My, i = row / g.My;
    const int fx = full_pos(i, g.hx, g.Mx, g.Nx), fy = full_pos(j, g.hy, g.My, g.Ny);
    const float2* ext = a.ext + ((long long)fx * g.Ny + fy) * g.Nzh;
    float2* cmp = a.cmp + (long long)row * g.Mzp;
    const float kx = a.k.kx[fx], ky = a.k.ky[fy];
    for (int k0 = lane; k0 < g.Mzp; k0 += 32 * LC_UNROLL) {
      float2 v[LC_UNROLL][3];
#pragma unroll
      for (int u = 0; u < LC_UNROLL; ++u) {
        const int k = k0 + 32 * u;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[u][c] = k < g.Mz ? ext[c * ce + k] : czero<float>();
      }
#pragma unroll
      for (int u = 0; u < LC_UNROLL; ++u) {
        const int k = k0 + 32 * u;
        if (k >= g.Mzp) break;
        if (a.partial && k < g.Mz) s.add(a, v[u], kx, ky, k);
#pragma unroll
        for (int c = 0; c < 3; ++c) cmp[c * cc + k] = v[u][c];
      }
    }
  }
  if (a.partial) s.store(a, red);
}

// float32 from 2^20 stored modes in rows of at least 128 points: 512^3 198 -> 171 us
// (2/3 box), 256^3 29.6 -> 27.5 and 86 -> 71 (general layout), 128 x 128 x 512 16.0 ->
// 14.8, general 128^3 14.0 -> 12.4; below, by rows: 128^3 6.5 -> 6.6, 64 x 64 x 1024 9.3 ->
// 10.7, 512 x 512 x 8 11 -> 31, 256 x 256 x 64 10.8 -> 13.1; float64 256^3 44.9 -> 45.9.
template <typename T> bool gather_by_rows(const Geom& g) {
  return sizeof(T) == 4 && g.Nz >= 128 && (long long)g.Mx * g.My * g.Mzp >= (1 << 20);
}
template <typename T> cudaError_t launch_gather(const GatherArgs<T>& a, int nblocks, cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    if (gather_by_rows<T>(a.g)) {
      k_gather_rows<<<nblocks, NT, 0, st>>>(a);
      return cudaGetLastError();
    }
  }
  k_gather<T><<<nblocks, NT, 0, st>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// scatter: compact -> reference layout (modes outside the compact set are 0)
// ---------------------------------------------------------------------------
// A thread per mode over the whole grid: successive warps write one run of memory,
// in whole lines.  With a warp per row (rows of Nz/2 + 1 entries start unaligned)
// the writes took 10 to 14% longer: 512^3 float32 2/3 box 411 against 469 us, general
// layout 565 against 634; 256^3 50 against 55; level at 128^3.
template <typename T>
__global__ void __launch_bounds__(NT) k_scatter(const V2<T>* __restrict__ cmp, V2<T>* __restrict__ ext, Geom g) {
  const long long nmodes = (long long)g.Nx * g.Ny * g.Nzh;
  const long long cc = (long long)g.Mx * g.My * g.Mzp;
  for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < nmodes; e += (long long)gridDim.x * NT) {
    const int k = (int)(e % g.Nzh);
    const long long r = e / g.Nzh;
    const int fy = (int)(r % g.Ny), fx = (int)(r / g.Ny);
    const int i = compact_row(fx, g.hx, g.Mx, g.Nx), j = compact_row(fy, g.hy, g.My, g.Ny);
    const bool kept = i >= 0 && j >= 0 && k < g.Mz;
    const long long m = kept ? ((long long)i * g.My + j) * g.Mzp + k : 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) ext[c * nmodes + e] = kept ? cmp[c * cc + m] : czero<T>();
  }
}

static int grid_for(long long n) {
  long long b = (n + NT - 1) / NT;
  return (int)(b < 8 * 148 ? (b < 1 ? 1 : b) : 8 * 148);
}

template <typename T> cudaError_t launch_scatter(const V2<T>* cmp, V2<T>* ext, const Geom& g, cudaStream_t st) {
  k_scatter<T><<<grid_for((long long)g.Nx * g.Ny * g.Nzh), NT, 0, st>>>(cmp, ext, g);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// flag modes outside the 2/3 box that are nonzero
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(NT) k_check_box(const V2<T>* __restrict__ ext, Geom g, int* flag) {
  const long long nmodes = (long long)g.Nx * g.Ny * g.Nzh;
  int found = 0;
  for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < nmodes; e += (long long)gridDim.x * NT) {
    const int k = (int)(e % g.Nzh);
    const long long r = e / g.Nzh;
    const int fy = (int)(r % g.Ny), fx = (int)(r / g.Ny);
    const bool in_box = abs(freq_of(fx, g.Nx)) <= g.cx && abs(freq_of(fy, g.Ny)) <= g.cy && k <= g.cz;
    if (!in_box) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const V2<T> v = ext[c * nmodes + e];
        found |= (v.x != T(0) || v.y != T(0));  // NaN compares unequal -> flagged
      }
    }
  }
  if (__syncthreads_or(found) && threadIdx.x == 0) atomicOr(flag, 1);
}

template <typename T>
__global__ void __launch_bounds__(NT) k_check_box_rows(const V2<T>* __restrict__ ext, Geom g, int* flag) {
  const long long ce = (long long)g.Nx * g.Ny * g.Nzh;
  const int lane = threadIdx.x & 31, nrows = g.Nx * g.Ny;
  int found = 0;
  for (int row = blockIdx.x * LC_WARPS + (threadIdx.x >> 5); row < nrows; row += gridDim.x * LC_WARPS) {
    const int fy = row % g.Ny, fx = row / g.Ny;
    const bool in_xy = abs(freq_of(fx, g.Nx)) <= g.cx && abs(freq_of(fy, g.Ny)) <= g.cy;
    const V2<T>* src = ext + (long long)row * g.Nzh;
    for (int k0 = (in_xy ? g.cz + 1 : 0) + lane; k0 < g.Nzh; k0 += 32 * LC_UNROLL) {
      V2<T> v[LC_UNROLL][3];
#pragma unroll
      for (int u = 0; u < LC_UNROLL; ++u) {
#pragma unroll
        for (int c = 0; c < 3; ++c) v[u][c] = k0 + 32 * u < g.Nzh ? src[c * ce + k0 + 32 * u] : czero<T>();
      }
#pragma unroll
      for (int u = 0; u < LC_UNROLL; ++u) {
#pragma unroll
        for (int c = 0; c < 3; ++c) found |= (v[u][c].x != T(0) || v[u][c].y != T(0));
      }
    }
  }
  if (__syncthreads_or(found) && threadIdx.x == 0) atomicOr(flag, 1);
}

// Rows of at least 64 points in float32 and 128 in float64, at least 4096 of them: by
// modes -> by rows, L2 flushed, 512^3 364 -> 213 us, 256^3 57 -> 39, 64 x 64 x 128 5.0 -> 4.2,
// 512 x 512 x 64 63 -> 56 (float64 74 -> 92), float64 128^3 12.7 -> 10.9 and 256^3 67 ->
// 68 (57 -> 53 with the state in L2); outside, 512 x 512 x 8 12.8 -> 48, 256 x 256 x 32 11 ->
// 15, 8 x 8 x 1024 2.6 -> 9.7, 32 x 32 x 256 3.3 -> 4.5.
template <typename T> bool check_by_rows(const Geom& g) {
  return g.Nz >= (sizeof(T) == 4 ? 64 : 128) && (long long)g.Nx * g.Ny >= 4096;
}
template <typename T> cudaError_t launch_check_box(const V2<T>* ext, const Geom& g, int* flag, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  if (check_by_rows<T>(g)) k_check_box_rows<T><<<grid_for((long long)g.Nx * g.Ny * 32), NT, 0, st>>>(ext, g, flag);
  else k_check_box<T><<<grid_for((long long)g.Nx * g.Ny * g.Nzh), NT, 0, st>>>(ext, g, flag);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// project(dealias(u)) in the reference layout (src/hit3d/grid.py:166-178)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(NT) k_dealias_project(const V2<T>* __restrict__ in, V2<T>* __restrict__ out, Geom g,
                                                        KTab<T> kt, int dd, int pp) {
  const long long nmodes = (long long)g.Nx * g.Ny * g.Nzh;
  for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < nmodes; e += (long long)gridDim.x * NT) {
    const int k = (int)(e % g.Nzh);
    const long long r = e / g.Nzh;
    const int fy = (int)(r % g.Ny), fx = (int)(r / g.Ny);
    V2<T> u[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = in[c * nmodes + e];
    if (dd && !in_dealias(g, fx, fy, k)) u[0] = u[1] = u[2] = czero<T>();
    if (pp) {
      const T kx = kt.kx[fx], ky = kt.ky[fy], kz = kt.kz[k];
      const T ik2 = inv_k2_of(k2_of(kx, ky, kz));
      V2<T> div;
      div.x = (kx * u[0].x + ky * u[1].x + kz * u[2].x) * ik2;
      div.y = (kx * u[0].y + ky * u[1].y + kz * u[2].y) * ik2;
      u[0] = csub(u[0], cscale(div, kx));
      u[1] = csub(u[1], cscale(div, ky));
      u[2] = csub(u[2], cscale(div, kz));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c * nmodes + e] = u[c];
  }
}

template <typename T>
cudaError_t launch_dealias_project(const V2<T>* in, V2<T>* out, const Geom& g, KTab<T> k, int dd, int pp, cudaStream_t st) {
  k_dealias_project<T><<<grid_for((long long)g.Nx * g.Ny * g.Nzh), NT, 0, st>>>(in, out, g, k, dd, pp);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// per-block spectral sums: shells (per component) and NSCAL scalars,
// compensated and in a fixed order (bit-identical from run to run)
// ---------------------------------------------------------------------------
struct KahanAcc {  // compensated running sum
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double x) {
    const double y = x - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const { return s - c; }
};

constexpr int MS_WARPS = 4;  // warps per k_mode_sums block

// A warp takes 32 consecutive kz modes of the up to four rows (+-kx, +-ky) at
// a time (the chunks are dealt to the warps of the grid in a fixed order):
// those rows share k2, the shell index and the weight, so their |u|^2 are
// added in registers first (12 loads in flight per lane) and everything after
// that -- weight, shell, scan, bins -- is done once for the four.  Along a row
// |k| and hence the shell index never decrease with kz, so the lanes of one
// shell form contiguous runs: a segmented shuffle scan in lane order gives
// each run's sum in its last lane, which adds it (Kahan) to the warp's own
// bins in shared memory; different runs have different shells, so no two
// lanes touch one bin.  E, Omega and the band energy are per-lane Kahan sums.
// At the end the warps' bins are added in warp order and the scalars by a
// fixed shuffle tree, so the result does not depend on scheduling.
// The scan's 35 shuffles and its float64 adds bound the kernel when they are
// done per row (256^3 float32: 165 us per launch with all four rows apart, 71
// together; 0.43 of HBM).
template <typename T>
__global__ void __launch_bounds__(MS_WARPS * 32) k_mode_sums(ModeSumArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nb3 = 3 * a.nshell;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* bs = reinterpret_cast<double*>(smem_raw);  // [warp][nb3] sums, then [warp][nb3] compensations
  double* bc = bs + MS_WARPS * nb3;
  __shared__ double red[32];
  for (int e = threadIdx.x; e < 2 * MS_WARPS * nb3; e += MS_WARPS * 32) bs[e] = 0.0;
  __syncthreads();
  const Geom& g = a.g;
  const int nck = (g.Mz + 31) / 32;
  // classes of rows with equal |kx| (|ky|): rows c and M - c, c = 0 .. M/2
  const int ncx = g.Mx / 2 + 1, ncy = g.My / 2 + 1;
  const long long nchunks = (long long)ncx * ncy * nck;
  double* wb = bs + warp * nb3;
  double* wc = bc + warp * nb3;
  KahanAcc sE, sO, sB;
  for (long long ch = (long long)blockIdx.x * MS_WARPS + warp; ch < nchunks; ch += (long long)gridDim.x * MS_WARPS) {
    const long long row = ch / nck;
    const int k = (int)(ch % nck) * 32 + lane;
    const int j = (int)(row % ncy), i = (int)(row / ncy);
    const bool on = k < g.Mz;
    const int fx = full_pos(i, g.hx, g.Mx, g.Nx), fy = full_pos(j, g.hy, g.My, g.Ny);
    const int i2 = g.Mx - i, j2 = g.My - j;  // the partner rows, where they are others
    const bool px = i > 0 && i2 != i, py = j > 0 && j2 != j;
    double e[3] = {0.0, 0.0, 0.0};
    int s = 0x7fffffff;  // lanes past the row: a key no real shell has
    if (on) {
      const V2<T>* p0 = a.u + (long long)i * a.c_x + (long long)j * a.c_y + k;
      const long long ox = (long long)(i2 - i) * a.c_x, oy = (long long)(j2 - j) * a.c_y;
      V2<T> v[4][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[0][c] = p0[c * a.c_c];
        v[1][c] = py ? p0[c * a.c_c + oy] : czero<T>();
        v[2][c] = px ? p0[c * a.c_c + ox] : czero<T>();
        v[3][c] = px && py ? p0[c * a.c_c + ox + oy] : czero<T>();
      }
      const T k2 = k2_of(a.k.kx[fx], a.k.ky[fy], a.k.kz[k]);
      const double w = herm_weight(g, k);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double q[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) q[r] = (double)v[r][c].x * v[r][c].x + (double)v[r][c].y * v[r][c].y;
        e[c] = w * ((q[0] + q[1]) + (q[2] + q[3]));
      }
      const double t = (e[0] + e[1]) + e[2];
      sE.add(t);
      sO.add((double)k2 * t);
      if (a.kmin2 <= k2 && k2 <= a.kmax2) sB.add(t);
      if (a.nshell > 0) {
        s = shell_of<T>(k2, a.k0);
        if (s < 0 || s >= a.nshell) s = 0x7ffffffe;  // not binned (a key of its own)
      }
    }
    if (a.nshell > 0) {
      // segmented inclusive scan over runs of equal s (contiguous in lane order)
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int so = __shfl_up_sync(0xffffffffu, s, d);
        double up[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) up[c] = __shfl_up_sync(0xffffffffu, e[c], d);
        if (lane >= d && so == s) {
#pragma unroll
          for (int c = 0; c < 3; ++c) e[c] += up[c];
        }
      }
      const int sn = __shfl_down_sync(0xffffffffu, s, 1);
      if (on && s < a.nshell && (lane == 31 || sn != s)) {  // last lane of its run
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int b = c * a.nshell + s;
          const double y = e[c] - wc[b];
          const double t = wb[b] + y;
          wc[b] = (t - wb[b]) - y;
          wb[b] = t;
        }
      }
      __syncwarp();
    }
  }
  const int NV = nb3 + NSCAL;
  double* out = a.partial + (long long)blockIdx.x * NV;
  double r = block_sum_f64(sE.value(), red);
  if (threadIdx.x == 0) out[nb3 + 0] = r;
  r = block_sum_f64(sO.value(), red);
  if (threadIdx.x == 0) out[nb3 + 1] = r;
  r = block_sum_f64(sB.value(), red);
  if (threadIdx.x == 0) out[nb3 + 2] = r;
  __syncthreads();
  for (int b = threadIdx.x; b < nb3; b += MS_WARPS * 32) {
    KahanAcc t;
#pragma unroll
    for (int w = 0; w < MS_WARPS; ++w) t.add(bs[w * nb3 + b] - bc[w * nb3 + b]);
    out[b] = t.value();
  }
}

template <typename T> size_t mode_sums_smem(int nshell) {
  return sizeof(double) * 2 * MS_WARPS * 3 * (size_t)(nshell > 0 ? nshell : 1);
}

template <typename T> cudaError_t launch_mode_sums(const ModeSumArgs<T>& a, int nblocks, cudaStream_t st) {
  const size_t smem = mode_sums_smem<T>(a.nshell);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_mode_sums<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_mode_sums<T><<<nblocks, MS_WARPS * 32, smem, st>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// out = u * c[shell(k)] (random_field's per-shell rescale, src/hit3d/fields.py:51-68)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(NT) k_shell_scale(const V2<T>* __restrict__ in, V2<T>* __restrict__ out, Geom g,
                                                    KTab<T> kt, T k0, const double* __restrict__ c, int smax) {
  const long long nmodes = (long long)g.Nx * g.Ny * g.Nzh;
  for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < nmodes; e += (long long)gridDim.x * NT) {
    const int k = (int)(e % g.Nzh);
    const long long r = e / g.Nzh;
    const int fy = (int)(r % g.Ny), fx = (int)(r / g.Ny);
    int s = shell_of<T>(k2_of(kt.kx[fx], kt.ky[fy], kt.kz[k]), k0);
    s = s < 0 ? 0 : (s > smax ? smax : s);  // out-of-range gathers clamp, as jnp indexing does
    const T f = (T)c[s];
#pragma unroll
    for (int q = 0; q < 3; ++q) out[q * nmodes + e] = cscale(in[q * nmodes + e], f);
  }
}

template <typename T>
cudaError_t launch_shell_scale(const V2<T>* in, V2<T>* out, const Geom& g, KTab<T> k, T k0, const double* c, int smax,
                               cudaStream_t st) {
  k_shell_scale<T><<<grid_for((long long)g.Nx * g.Ny * g.Nzh), NT, 0, st>>>(in, out, g, k, k0, c, smax);
  return cudaGetLastError();
}
template cudaError_t launch_shell_scale<float>(const float2*, float2*, const Geom&, KTab<float>, float, const double*, int, cudaStream_t);
template cudaError_t launch_shell_scale<double>(const double2*, double2*, const Geom&, KTab<double>, double, const double*, int, cudaStream_t);

// ---------------------------------------------------------------------------
// finalisers
// ---------------------------------------------------------------------------
struct Kahan {
  double s = 0.0, c = 0.0;
  __device__ void add(double x) {
    const double y = x - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

__device__ __forceinline__ double forcing_coef(int forcing, double E, double Om, double twoEb, double nu, double eps,
                                               double Et, double tau, double tiny, double A) {
  if (forcing == 1) return A;
  if (forcing == 2) return twoEb > tiny ? eps / twoEb : 0.0;
  if (forcing == 3) {
    const double relax = (tau > 0.0 && isfinite(tau)) ? (E - Et) / tau : 0.0;
    return E > 0.0 ? (2.0 * nu * Om - relax) / (2.0 * E) : 0.0;
  }
  return 0.0;
}

// One 1024-thread block: thread t Kahan-sums rows t, t + 1024, ... of the
// three columns in order, issuing the loads of CB rows before adding them (the
// row chain is latency-bound otherwise), then fixed shuffle trees combine the
// threads.
constexpr int COEF_THREADS = 1024;
__global__ void __launch_bounds__(COEF_THREADS) k_finalize_coef(CoefArgs a) {
  __shared__ double red[96];
  pdl_wait();
  pdl_trigger();
  constexpr int CB = 4;
  Kahan k0, k1, k2;
  for (int b0 = threadIdx.x; b0 < a.nblocks; b0 += CB * COEF_THREADS) {
    double v[CB][3];
#pragma unroll
    for (int i = 0; i < CB; ++i) {
      const int b = b0 + i * COEF_THREADS;
#pragma unroll
      for (int c = 0; c < 3; ++c) v[i][c] = b < a.nblocks ? a.partial[3 * (long long)b + c] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < CB; ++i) {
      if (b0 + i * COEF_THREADS < a.nblocks) {
        k0.add(v[i][0]);
        k1.add(v[i][1]);
        k2.add(v[i][2]);
      }
    }
  }
  double S0 = k0.s - k0.c, S1 = k1.s - k1.c, S2 = k2.s - k2.c;
  block_sum3_f64(S0, S1, S2, red);
  if (threadIdx.x == 0) {
    const double E = S0 / (2.0 * a.ntot2), Om = S1 / (2.0 * a.ntot2), twoEb = S2 / a.ntot2;
    a.coef[0] = forcing_coef(a.forcing, E, Om, twoEb, a.nu, a.eps, a.E_target, a.tau, a.tiny, 0.0);
    a.coef[1] = E;
    a.coef[2] = Om;
    a.coef[3] = twoEb;
  }
}

cudaError_t launch_finalize_coef(const CoefArgs& a, cudaStream_t st) {
  return launch_pdl(k_finalize_coef, 1, COEF_THREADS, 0, st, a);
}

// Column sums of partial[nblocks][nvals]: a block takes 32 columns (one per
// lane, 256-byte row segments), warp w Kahan-sums rows w, w + FS_WARPS, ... in
// order with FS_BATCH loads in flight, and the warps' sums are Kahan-added in
// warp order.  What bounds it is the latency of one thread's row chain: with a
// thread per column walking all rows one load at a time, 1184 rows x 6 columns
// took 136 us (740 x 675: 104 us); here a chain is 1/32 of the rows and its
// loads overlap.
constexpr int FS_WARPS = 32, FS_BATCH = 8;
__global__ void __launch_bounds__(FS_WARPS * 32) k_finalize_sums(SumArgs a) {
  __shared__ double part[FS_WARPS][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + lane;
  Kahan k;
  if (v < a.nvals) {
    for (int b0 = warp; b0 < a.nblocks; b0 += FS_WARPS * FS_BATCH) {
      double x[FS_BATCH];
#pragma unroll
      for (int i = 0; i < FS_BATCH; ++i) {
        const int b = b0 + i * FS_WARPS;
        x[i] = b < a.nblocks ? a.partial[(long long)b * a.nvals + v] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < FS_BATCH; ++i)
        if (b0 + i * FS_WARPS < a.nblocks) k.add(x[i]);
    }
  }
  part[warp][lane] = k.s - k.c;
  __syncthreads();
  if (warp == 0 && v < a.nvals) {
    Kahan t;
#pragma unroll
    for (int w = 0; w < FS_WARPS; ++w) t.add(part[w][lane]);
    a.sums[v] = t.s - t.c;
  }
}

cudaError_t launch_finalize_sums(const SumArgs& a, cudaStream_t st) {
  k_finalize_sums<<<(a.nvals + 31) / 32, FS_WARPS * 32, 0, st>>>(a);
  return cudaGetLastError();
}

__global__ void k_finalize_budget(BudgetArgs a) {
  const int ns = a.nshell;
  const double inv = 1.0 / (2.0 * a.ntot2);
  for (int s = 1 + threadIdx.x; s < ns; s += blockDim.x) {
    const double c0 = a.sums[s] * inv, c1 = a.sums[ns + s] * inv, c2 = a.sums[2 * ns + s] * inv;
    if (a.spec) a.spec[s - 1] = c0 + c1 + c2;
    if (a.comp) {
      a.comp[s - 1] = c0;
      a.comp[(ns - 1) + s - 1] = c1;
      a.comp[2 * (ns - 1) + s - 1] = c2;
    }
  }
  if (threadIdx.x == 0 && a.budget) {
    const double* sc = a.sums + 3 * ns;
    const double E = sc[0] * inv, Om = sc[1] * inv, twoEb = sc[2] / a.ntot2;
    const double cf = forcing_coef(a.forcing, E, Om, twoEb, a.nu, a.eps, a.E_target, a.tau, a.tiny, a.A);
    double P = 0.0;
    if (a.forcing == 1 || a.forcing == 3) P = cf * 2.0 * E;
    else if (a.forcing == 2) P = twoEb > a.tiny ? a.eps : 0.0;
    a.budget[0] = E;
    a.budget[1] = 2.0 * a.nu * Om;
    a.budget[2] = P;
    a.budget[3] = Om;
  }
}

cudaError_t launch_finalize_budget(const BudgetArgs& a, cudaStream_t st) {
  k_finalize_budget<<<1, NT, 0, st>>>(a);
  return cudaGetLastError();
}

template cudaError_t launch_gather<float>(const GatherArgs<float>&, int, cudaStream_t);
template cudaError_t launch_gather<double>(const GatherArgs<double>&, int, cudaStream_t);
template cudaError_t launch_scatter<float>(const float2*, float2*, const Geom&, cudaStream_t);
template cudaError_t launch_scatter<double>(const double2*, double2*, const Geom&, cudaStream_t);
template cudaError_t launch_check_box<float>(const float2*, const Geom&, int*, cudaStream_t);
template cudaError_t launch_check_box<double>(const double2*, const Geom&, int*, cudaStream_t);
template cudaError_t launch_dealias_project<float>(const float2*, float2*, const Geom&, KTab<float>, int, int, cudaStream_t);
template cudaError_t launch_dealias_project<double>(const double2*, double2*, const Geom&, KTab<double>, int, int, cudaStream_t);
template cudaError_t launch_mode_sums<float>(const ModeSumArgs<float>&, int, cudaStream_t);
template cudaError_t launch_mode_sums<double>(const ModeSumArgs<double>&, int, cudaStream_t);

}  // namespace hit
