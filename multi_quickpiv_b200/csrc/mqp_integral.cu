// sm_100a kernels of the FP64 integral images and volumes the normalised
// similarities read.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mqp_finish.cuh"
#include "mqp_internal.h"

namespace mqp {

// ---------------------------------------------------------------------------
// integral images (integralArraySQ!, src/utils/common_ops.jl:142-180, built
// once per image instead of once per search window)
// ---------------------------------------------------------------------------
// pass 1: one warp per image column, prefix sum down the column (dim 1,
// contiguous) with warp scans; writes rows 1..H of out column c+1 and the
// zero first row.
// blockIdx.y selects one of a batch of planes (the z slices of a volume):
// input plane z starts at img + z*in_plane, its output at out + z*out_plane.
// Output columns [cb, ce) of the (W+1)-column integral.
//
// A warp takes COLG groups of 32 rows at a time: their loads are issued
// together, their shuffle scans are independent chains, and only one add per
// group carries the running sum on (the total of a group is its own scan's
// last value, so every sum is formed in the order of one group after the
// other).  One group at a time the pass was bound by the latency of that chain.
constexpr int COLG = 8;

template <typename T, bool SQ>
__global__ void __launch_bounds__(256) integral_cols_kernel(const T* __restrict__ img, int H, int W,
                                                            double* __restrict__ out, long long in_plane,
                                                            long long out_plane, int cb, int ce) {
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long ld = (long long)H + 1;
  img += in_plane * blockIdx.y;
  out += out_plane * blockIdx.y;
  for (int c = cb + blockIdx.x * warps + (threadIdx.x >> 5); c < ce; c += gridDim.x * warps) {
    double* o = out + ld * c;
    if (c == 0) {
      for (int r = lane; r <= H; r += 32) o[r] = 0.0;
      continue;
    }
    const T* col = img + (long long)H * (c - 1);
    if (lane == 0) o[0] = 0.0;
    double carry = 0.0;
    for (int r0 = 0; r0 < H; r0 += 32 * COLG) {
      T x[COLG];
#pragma unroll
      for (int g = 0; g < COLG; ++g) {
        const int r = r0 + 32 * g + lane;
        x[g] = r < H ? col[r] : T(0);
      }
      double v[COLG];
#pragma unroll
      for (int g = 0; g < COLG; ++g) {
        v[g] = (double)x[g];
        if (SQ) v[g] = v[g] * v[g];
      }
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
        for (int g = 0; g < COLG; ++g) {
          const double t = __shfl_up_sync(0xffffffffu, v[g], off);
          if (lane >= off) v[g] += t;
        }
      }
#pragma unroll
      for (int g = 0; g < COLG; ++g) {
        const int r = r0 + 32 * g + lane;
        const double total = __shfl_sync(0xffffffffu, v[g], 31);
        v[g] += carry;
        if (r < H) o[r + 1] = v[g];
        carry = total + carry;
      }
    }
  }
}

// pass 2: running sums across columns (dim 2) in chunks of ICHUNK columns:
// thread (row r, chunk k) scans its chunk in place and records the chunk
// total; consecutive threads take consecutive rows, so every step is a
// coalesced column segment.
constexpr int ICHUNK = 64;
// values a thread of the row and z passes loads before it uses any: the
// stores in between would otherwise hold back the next load for a round trip
constexpr int IBATCH = 16;

__global__ void integral_rows_chunk_kernel(int H, int W, double* __restrict__ out, double* __restrict__ totals,
                                           long long out_plane, long long tot_plane, int k0) {
  const long long ld = (long long)H + 1;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y + k0;
  if (r > H) return;
  out += out_plane * blockIdx.z;
  totals += tot_plane * blockIdx.z;
  const int c0 = 1 + k * ICHUNK;
  const int c1 = c0 + ICHUNK <= W + 1 ? c0 + ICHUNK : W + 1;
  double acc = 0.0;
  int c = c0;
  for (; c + IBATCH <= c1; c += IBATCH) {
    double v[IBATCH];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) v[t] = out[r + ld * (c + t)];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) {
      acc += v[t];
      out[r + ld * (c + t)] = acc;
    }
  }
  for (; c < c1; ++c) {
    acc += out[r + ld * c];
    out[r + ld * c] = acc;
  }
  totals[r + ld * k] = acc;
}

// pass 3a: per row, the running sums of the chunk totals,
// offs[k] = ((t_0 + t_1) + ...) + t_{k-1}, for chunks k in [k0, k1), k0 >= 1,
// continuing from offs[k0 - 1] (left by the earlier chunks).  offs lives
// tot_plane / 2 after the totals of its plane.
__global__ void integral_rows_prefix_kernel(int H, double* __restrict__ totals, long long tot_plane, int k0, int k1) {
  const long long ld = (long long)H + 1;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > H) return;
  totals += tot_plane * blockIdx.z;
  double* offs = totals + tot_plane / 2;
  double off = k0 > 1 ? offs[r + ld * (k0 - 1)] : 0.0;
  for (int k = k0; k < k1; ++k) {
    off = (k > 1 ? off : 0.0) + totals[r + ld * (k - 1)];
    offs[r + ld * k] = off;
  }
}

// pass 3b: every chunk k > 0 adds the sum of the totals of chunks 0..k-1
// (chunks k0 + blockIdx.y, k0 >= 1): read from pass 3a's running sums, or
// (few chunks, no pass 3a) summed here in the same order.
__global__ void integral_rows_offset_kernel(int H, int W, double* __restrict__ out,
                                            const double* __restrict__ totals, long long out_plane,
                                            long long tot_plane, int k0, int prefixed) {
  const long long ld = (long long)H + 1;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y + k0;
  if (r > H) return;
  out += out_plane * blockIdx.z;
  totals += tot_plane * blockIdx.z;
  double off = 0.0;
  if (prefixed) {
    off = totals[tot_plane / 2 + r + ld * k];
  } else {
    for (int q = 0; q < k; ++q) off += totals[r + ld * q];
  }
  const int c0 = 1 + k * ICHUNK;
  const int c1 = c0 + ICHUNK <= W + 1 ? c0 + ICHUNK : W + 1;
  int c = c0;
  for (; c + IBATCH <= c1; c += IBATCH) {
    double v[IBATCH];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) v[t] = out[r + ld * (c + t)];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) out[r + ld * (c + t)] = v[t] + off;
  }
  for (; c < c1; ++c) out[r + ld * c] += off;
}

// pass 4 (volumes): running sums along dim 3, one thread per (row, column)
// walking the planes; consecutive threads take consecutive rows.
__global__ void integral_zscan_kernel(long long plane, int D, double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= plane) return;
  double acc = 0.0;
  int z = 1;
  for (; z + IBATCH <= D + 1; z += IBATCH) {
    double v[IBATCH];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) v[t] = out[plane * (z + t) + i];
#pragma unroll
    for (int t = 0; t < IBATCH; ++t) {
      acc += v[t];
      out[plane * (z + t) + i] = acc;
    }
  }
  for (; z <= D; ++z) {
    double* p = out + plane * z + i;
    acc += *p;
    *p = acc;
  }
}

// 2D exclusive-prefix integrals of `planes` consecutive H x W planes of img,
// plane z written to out + z*out_plane: the integral columns that image
// columns [x0, x1) complete (x0 a multiple of 64, x1 one or W), after those
// of image columns < x0.  Piece by piece or at once, every value comes out
// of the same sums in the same order.
static cudaError_t integral_planes(const void* img, int dtype, int H, int W, int planes, bool square, double* out,
                                   long long out_plane, double* scratch, cudaStream_t s, int x0 = 0, int x1 = -1) {
  if (x1 < 0) x1 = W;
  if (x0 % ICHUNK != 0 || x1 <= x0 || x1 > W || (x1 % ICHUNK != 0 && x1 != W)) return cudaErrorInvalidValue;
  const int threads = 256;
  const int cb = x0 == 0 ? 0 : x0 + 1, ce = x1 + 1;  // integral column c sums image columns < c
  const int blocks = (ce - cb + 7) / 8 < 4096 ? (ce - cb + 7) / 8 : 4096;
  const long long in_plane = (long long)H * W;
  const dim3 gc(blocks, planes);
  if (dtype == 0) {
    if (square) integral_cols_kernel<float, true><<<gc, threads, 0, s>>>((const float*)img, H, W, out, in_plane, out_plane, cb, ce);
    else integral_cols_kernel<float, false><<<gc, threads, 0, s>>>((const float*)img, H, W, out, in_plane, out_plane, cb, ce);
  } else {
    if (square) integral_cols_kernel<double, true><<<gc, threads, 0, s>>>((const double*)img, H, W, out, in_plane, out_plane, cb, ce);
    else integral_cols_kernel<double, false><<<gc, threads, 0, s>>>((const double*)img, H, W, out, in_plane, out_plane, cb, ce);
  }
  const int chunks = (W + ICHUNK - 1) / ICHUNK;
  const int k0 = x0 / ICHUNK, k1 = (x1 + ICHUNK - 1) / ICHUNK;  // row chunks of this piece
  // per plane: the chunk totals, then their running sums
  const long long tot_plane = 2LL * (H + 1) * (chunks + 1);
  const dim3 g1((H + 1 + 127) / 128, k1 - k0, planes);
  integral_rows_chunk_kernel<<<g1, 128, 0, s>>>(H, W, out, scratch, out_plane, tot_plane, k0);
  const int ko = k0 > 1 ? k0 : 1;
  if (k1 > ko) {
    // wide images: running sums first (linear work); up to 32 chunks the
    // offsets sum their few totals directly (one launch fewer)
    const int prefixed = chunks > 32;
    if (prefixed) {
      const dim3 gp((H + 1 + 127) / 128, 1, planes);
      integral_rows_prefix_kernel<<<gp, 128, 0, s>>>(H, scratch, tot_plane, ko, k1);
    }
    const dim3 g2((H + 1 + 127) / 128, k1 - ko, planes);
    integral_rows_offset_kernel<<<g2, 128, 0, s>>>(H, W, out, scratch, out_plane, tot_plane, ko, prefixed);
  }
  return cudaGetLastError();
}

cudaError_t launch_integral2d(const void* img, int dtype, int H, int W, bool square, double* out,
                              double* scratch, cudaStream_t s) {
  return integral_planes(img, dtype, H, W, 1, square, out, 0, scratch, s);
}

cudaError_t launch_integral2d_cols(const void* img, int dtype, int H, int W, int x0, int x1, bool square,
                                   double* out, double* scratch, cudaStream_t s) {
  return integral_planes(img, dtype, H, W, 1, square, out, 0, scratch, s, x0, x1);
}

cudaError_t launch_integral3d(const void* img, int dtype, int H, int W, int D, bool square, double* out,
                              double* scratch, cudaStream_t s) {
  const long long plane = (long long)(H + 1) * (W + 1);
  cudaError_t e = cudaMemsetAsync(out, 0, (size_t)plane * sizeof(double), s);
  if (e != cudaSuccess) return e;
  // planes are independent in the 2D passes; the grid's y/z extent bounds a batch
  for (int z0 = 0; z0 < D; z0 += 65535) {
    const int nz = D - z0 < 65535 ? D - z0 : 65535;
    const char* src = (const char*)img + (size_t)z0 * H * W * (dtype == 0 ? 4 : 8);
    e = integral_planes(src, dtype, H, W, nz, square, out + plane * (1 + z0), plane, scratch, s);
    if (e != cudaSuccess) return e;
  }
  integral_zscan_kernel<<<(unsigned)((plane + 255) / 256), 256, 0, s>>>(plane, D, out);
  return cudaGetLastError();
}

size_t integral2d_scratch_bytes(int H, int W) {  // chunk totals and their running sums
  return 2 * (size_t)(H + 1) * (size_t)((W + ICHUNK - 1) / ICHUNK + 1) * sizeof(double);
}

size_t integral3d_scratch_bytes(int H, int W, int D) {
  return integral2d_scratch_bytes(H, W) * (size_t)(D < 65535 ? D : 65535);
}

// ---------------------------------------------------------------------------
// window-sum map of a pass (mqp_finish.cuh) from the integral image of img2^2
// ---------------------------------------------------------------------------
// One thread per row of the map and WMAP columns: consecutive threads read
// and write consecutive rows.
constexpr int WMAP = 4;

__device__ __forceinline__ void window_sums(const double* __restrict__ II, long long ld, int W, int IS2, int SM2, int r0,
                                            int r1, int j0, int cols, double (&S)[WMAP]) {
  double a11[WMAP], a10[WMAP], a01[WMAP], a00[WMAP];
#pragma unroll
  for (int t = 0; t < WMAP; ++t) {
    const int j = j0 + t - SM2;
    const int c0 = j > 0 ? j : 0, c1 = j + IS2 < W ? j + IS2 : W;
    const bool any = j0 + t < cols && r1 > r0 && c1 > c0;
    const double* A1 = II + ld * c1;
    const double* A0 = II + ld * c0;
    a11[t] = any ? A1[r1] : 0.0;
    a10[t] = any ? A1[r0] : 0.0;
    a01[t] = any ? A0[r1] : 0.0;
    a00[t] = any ? A0[r0] : 0.0;
  }
#pragma unroll
  for (int t = 0; t < WMAP; ++t) S[t] = (a11[t] - a10[t]) - (a01[t] - a00[t]);  // box_sum's order
}

// NSQECC: ws (and wd) from II2; ZNCC: wz from II2 and II1 (IIg2 and IIg).
__global__ void __launch_bounds__(256) window_map_kernel(const double* __restrict__ II2, const double* __restrict__ II1,
                                                         int H, int W, int IS1, int IS2, int SM1, int SM2,
                                                         WindowMap m, int cols, int col0) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m.ldw) return;
  const long long ld = (long long)H + 1;
  const int i = k - SM1;
  const int r0 = i > 0 ? i : 0, r1 = i + IS1 < H ? i + IS1 : H;
  const int j0 = col0 + (int)blockIdx.y * WMAP;
  double S2[WMAP], S1[WMAP];
  window_sums(II2, ld, W, IS2, SM2, r0, r1, j0, cols, S2);
  if (m.wz) window_sums(II1, ld, W, IS2, SM2, r0, r1, j0, cols, S1);
#pragma unroll
  for (int t = 0; t < WMAP; ++t) {
    if (j0 + t < cols) {
      const long long at = k + (long long)m.ldw * (j0 + t);
      if (m.wz) {
        m.wz[at] = make_double2(S2[t], S1[t]);
      } else {
        const float s = (float)S2[t];
        m.ws[at] = make_float2(s, sqrtf(s));
        if (m.wd) m.wd[at] = S2[t];
      }
    }
  }
}

WindowMap window_map(int H, int W, int IS1, int IS2, int SM1, int SM2, int alg, bool SN, void* base) {
  WindowMap m;
  m.ldw = winmap_ld(H, IS1, SM1);
  m.cols = winmap_ld(W, IS2, SM2);
  const size_t n = (size_t)m.ldw * (size_t)m.cols;
  if (alg == ALG_ZNCC) {
    m.wz = (double2*)base;
    m.bytes = n * sizeof(double2);
  } else {
    m.ws = (float2*)base;
    m.bytes = n * sizeof(float2);
    if (SN) {
      m.wd = (double*)((char*)base + m.bytes);
      m.bytes += n * sizeof(double);
    }
  }
  return m;
}

cudaError_t launch_window_map(const double* II2, const double* II1, int H, int W, int IS1, int IS2, int SM1, int SM2,
                              const WindowMap& m, int m0, int m1, cudaStream_t s) {
  const int threads = m.ldw < 256 ? (m.ldw + 31) / 32 * 32 : 256;
  for (int c0 = m0; c0 < m1; c0 += 65535 * WMAP) {
    const int n = m1 - c0 < 65535 * WMAP ? m1 - c0 : 65535 * WMAP;
    const dim3 grid((m.ldw + threads - 1) / threads, (n + WMAP - 1) / WMAP);
    window_map_kernel<<<grid, threads, 0, s>>>(II2, II1, H, W, IS1, IS2, SM1, SM2, m, c0 + n, c0);
  }
  return cudaGetLastError();
}

}  // namespace mqp
