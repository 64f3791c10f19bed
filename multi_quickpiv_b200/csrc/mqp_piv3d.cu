// sm_100a kernels of the 3D path (see mqp_piv3d.cuh): K3a (r2c along dim 3),
// K3b (complex 2D correlation per k3 slab), K3c (inverse along k3, similarity,
// peak, Gaussian fit, SN), launched chunk by chunk over the vector field.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "mqp_finish3.cuh"
#include "mqp_internal.h"

namespace mqp {

namespace {

constexpr int K3A_THREADS = 256;

__device__ __forceinline__ double warp_sum3(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double warp_max3(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ double warp_nmax3(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = nmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// Blocks (part, IA): each part walks its contiguous share of the IA's lines.
// Pass 0 leaves the part's skip maxima and sumF2 in apart; part 0 records the
// ZNCC means, and k3a_merge_kernel completes the state.
// Two blocks per SM (16 warps): registers capped at 128 (a few bytes of
// spill at length 64) instead of one 147-register block.
template <int N, bool FPRUNE, int ALG, typename T>
__global__ void __launch_bounds__(K3A_THREADS, 2) k3a_kernel(Piv3dArgs a, int pass) {
  constexpr int PARTS = k3a_parts(N);
  const int part = blockIdx.x;
  const long long ci = blockIdx.y;
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  IA3State s;
  if (pass == 0) {
    ia3_means<ALG>(a, g, s.meanF, s.meanG);
    s.sumF2 = 0.0;
    s.skip = 0;
  } else {
    s = a.state[ci];
  }
  double vmax = -INFINITY, mmax = -INFINITY, sumsq = 0.0;
  const int nl = k3a_lines(a, g);
  const int l0 = (int)((long long)nl * part / PARTS), l1 = (int)((long long)nl * (part + 1) / PARTS);
  for (int line = l0 + threadIdx.x; line < l1; line += K3A_THREADS)
    k3a_line<N, FPRUNE, T, ALG>(a, g, s, pass, ci, line, vmax, mmax, sumsq);
  if (pass != 0) return;
  __shared__ double red[3][K3A_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  vmax = warp_max3(vmax);
  mmax = warp_max3(mmax);
  sumsq = warp_sum3(sumsq);
  if (lane == 0) {
    red[0][warp] = vmax;
    red[1][warp] = mmax;
    red[2][warp] = sumsq;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < K3A_THREADS / 32; ++w) {
      vmax = fmax(vmax, red[0][w]);
      mmax = fmax(mmax, red[1][w]);
      sumsq += red[2][w];
    }
    a.apart[ci * PARTS + part] = ReducePart3{vmax, mmax, sumsq};
    if (part == 0) a.state[ci] = s;
  }
}

// One thread per IA: its K3a parts in part order -> sumF2 and the skip test.
template <int N, int ALG>
__global__ void k3a_merge_kernel(Piv3dArgs a, long long n) {
  constexpr int PARTS = k3a_parts(N);
  const long long ci = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= n) return;
  const ReducePart3* p = a.apart + ci * PARTS;
  double vmax = p[0].vmax, mmax = p[0].mmax, sumsq = p[0].sumsq;
  for (int k = 1; k < PARTS; ++k) {
    vmax = fmax(vmax, p[k].vmax);
    mmax = fmax(mmax, p[k].mmax);
    sumsq += p[k].sumsq;
  }
  IA3State s = a.state[ci];
  s.sumF2 = sumsq;
  s.skip = skip_test3(a, ALG, vmax, mmax) ? 1 : 0;
  a.state[ci] = s;
}

// z-spectra of whole image layers: without a predictor every IA of one
// vector-field z index reads the same z window, so a line's r2c along dim 3
// (k3a_line) serves every IA that covers it (16 at step 16 and windows of 64).
// Thread per line; blockIdx.z = 2 layer + (0: G, 1: F).  FFTCC and NSQECC (ZNCC
// subtracts each IA's own mean first).
template <int N, bool FPRUNE, typename T>
__global__ void __launch_bounds__(256) k3s_lines_kernel(Piv3dArgs a) {
  constexpr int M = N / 2;
  const long long HW = (long long)a.H * a.W;
  const int x1 = blockIdx.x * blockDim.x + threadIdx.x, x2 = blockIdx.y, l = blockIdx.z >> 1;
  if (x1 >= a.H) return;
  const IAGeom3 g = ia_geom3(a, (long long)a.vf[0] * a.vf[1] * (a.l0 + l));
  const long long at = x1 + (long long)a.H * x2;
  float2* out = ((blockIdx.z & 1) ? a.Fs : a.Gs) + (x1 + a.pitch * x2 + a.lstride * l);
  float2 z[M];
  if (blockIdx.z & 1) {
    const T* p = reinterpret_cast<const T*>(a.img1) + (at + HW * g.ir[2]);
    constexpr int FLIM = Lay3<N, FPRUNE>::NF;
#pragma unroll
    for (int n = 0; n < M; ++n) {
      const int u = 2 * n, v = 2 * n + 1;
      z[n] = make_float2(0.f, 0.f);
      if (u < FLIM) z[n].x = (float)ldg_px<T>(p, HW * min(u, a.IS[2] - 1));
      if (v < FLIM) z[n].y = (float)ldg_px<T>(p, HW * min(v, a.IS[2] - 1));
    }
#pragma unroll
    for (int n = 0; n < M; ++n) {
      if (2 * n >= a.IS[2]) z[n].x = 0.f;
      if (2 * n + 1 >= a.IS[2]) z[n].y = 0.f;
    }
    r2c_line_store<N, FPRUNE ? M / 2 : M>(z, out, a.zplane);
  } else {
    const T* p = reinterpret_cast<const T*>(a.img2) + (at + HW * g.g0[2]);
    const int zl = g.lo[2], zh = g.hi[2];
#pragma unroll
    for (int n = 0; n < M; ++n) {
      const int u = 2 * n, v = 2 * n + 1;
      z[n] = make_float2((float)ldg_px<T>(p, HW * min(max(u, zl), zh - 1)), (float)ldg_px<T>(p, HW * min(max(v, zl), zh - 1)));
    }
#pragma unroll
    for (int n = 0; n < M; ++n) {
      if (2 * n < zl || 2 * n >= zh) z[n].x = 0.f;
      if (2 * n + 1 < zl || 2 * n + 1 >= zh) z[n].y = 0.f;
    }
    r2c_line_store<N, M>(z, out, a.zplane);
  }
}

// With shared z-spectra: an IA's skip maximum and sumF2, a block per IA.  The FP64
// sum adds lines where k3a_kernel adds pixels over a thread's lines, so the two
// sumF2 agree to FP64 rounding; the similarities' FP32 quotients rarely show it.
template <typename T, int ALG>
__global__ void __launch_bounds__(K3A_THREADS) k3s_state_kernel(Piv3dArgs a) {
  const long long ci = blockIdx.x;
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  const long long HW = (long long)a.H * a.W;
  double vmax = -INFINITY, sumsq = 0.0;
  const int nl = a.IS[0] * a.IS[1];
  constexpr int LB = 4;  // lines a thread sums at once: as many independent chains
  for (int l0 = threadIdx.x; l0 < nl; l0 += LB * K3A_THREADS) {
    const T* p[LB];
    bool in[LB];
    double sq[LB];
#pragma unroll
    for (int k = 0; k < LB; ++k) {
      const int line = l0 + k * K3A_THREADS;
      in[k] = line < nl;
      const int x1 = in[k] ? line % a.IS[0] : 0, x2 = in[k] ? line / a.IS[0] : 0;
      p[k] = reinterpret_cast<const T*>(a.img1) +
             ((long long)(g.ir[0] + x1) + (long long)a.H * ((long long)(g.ir[1] + x2) + (long long)a.W * g.ir[2]));
      sq[k] = 0.0;
    }
#pragma unroll 4
    for (int x = 0; x < a.IS[2]; ++x) {
#pragma unroll
      for (int k = 0; k < LB; ++k) {
        const double r = (double)ldg_px<T>(p[k], HW * x);
        vmax = in[k] && r > vmax ? r : vmax;
        sq[k] += r * r;
      }
    }
#pragma unroll
    for (int k = 0; k < LB; ++k) sumsq += in[k] ? sq[k] : 0.0;
  }
  __shared__ double red[2][K3A_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  vmax = warp_max3(vmax);
  sumsq = warp_sum3(sumsq);
  if (lane == 0) {
    red[0][warp] = vmax;
    red[1][warp] = sumsq;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < K3A_THREADS / 32; ++w) {
      vmax = fmax(vmax, red[0][w]);
      sumsq += red[1][w];
    }
    a.state[ci] = IA3State{sumsq, 0.0, 0.0, skip_test3(a, ALG, vmax, vmax) ? 1 : 0, 0};
  }
}

// One block of 2N threads (a pair per line) per (k3, IA) slab.
template <int N, bool FPRUNE, bool SHARED>
__global__ void __launch_bounds__(2 * N) k3b_kernel(Piv3dArgs a, float2* C) {
  using L = Lay3<N, FPRUNE>;
  constexpr int M = N / 2;
  extern __shared__ float2 sm[];
  const int k3 = blockIdx.x;
  const long long ci = blockIdx.y;
  if (a.state[ci].skip) return;
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  const int P1 = 2 * a.SM[0] + 1, P2 = 2 * a.SM[1] + 1;
  float2* S = sm;
  float2* SF = sm + N * L::SSTR;
  const int t = threadIdx.x % N, h = threadIdx.x / N;
  if (SHARED) k3b_rows_shared<N, FPRUNE>(a, g, k3, t, h, S, SF);
  else k3b_rows<N, FPRUNE>(a, g, ci, k3, t, h, S, SF);
  __syncthreads();
  {
    float2 y[M];
    k3b_cols_g<N, FPRUNE>(t, h, S, y);
    __syncthreads();
    k3b_park<N, FPRUNE>(t, h, S, y);
  }
  __syncthreads();
  {
    float2 p[M];
    k3b_cols_f<N, FPRUNE>(t, h, S, SF, p);
    __syncthreads();
    k3b_x1<N, FPRUNE>(t, h, p, S, P1);
    __syncthreads();
    float2 o[M];
    k3b_x2<N, FPRUNE>(t, h, S, o, P1, p);
    __syncthreads();
    k3b_x3<N, FPRUNE>(t, h, P1, o, S);
  }
  __syncthreads();
  {
    // the 2 P1 half rows go to consecutive threads: at 33 lags three warps
    // work where (t, h) would take all four for two of their lanes
    const int t2 = threadIdx.x % P1, h2 = threadIdx.x / P1;  // P1 <= N
    const int tr = h2 < 2 ? t2 : P1;
    float2 u[M];
    k3b_r2a<N, FPRUNE>(tr, h2, P1, S, u);
    __syncthreads();
    k3b_r2b<N, FPRUNE>(tr, h2, P1, u, S, P2);
    __syncthreads();
    k3b_r2c<N, FPRUNE>(ci, k3, tr, h2, P1, P2, S, C, u);
  }
}

// Blocks (part, IA): each part walks its contiguous share of the lag pairs;
// the part's peak / SN accumulators go to cpart, and k3c_merge_kernel
// finishes the IA.
template <int N, int ALG>
__global__ void __launch_bounds__(K3C_THREADS) k3c_kernel(Piv3dArgs a) {
  const int part = blockIdx.x, parts = gridDim.x;
  const long long ci = blockIdx.y;
  const int P1 = 2 * a.SM[0] + 1, P2 = 2 * a.SM[1] + 1, P3 = 2 * a.SM[2] + 1;
  const int q0 = P1 * P2 * part / parts, q1 = P1 * P2 * (part + 1) / parts;
  const IA3State s = a.state[ci];
  if (s.skip) {
    if (a.planes) {
      const long long vol = (long long)P1 * P2 * P3;
      double* dst = a.planes + (a.ia_begin + ci - a.planes_begin) * vol;
      for (int q = q0 + threadIdx.x; q < q1; q += K3C_THREADS)
        for (int s3 = 0; s3 < P3; ++s3) dst[q + (long long)P1 * P2 * s3] = 0.0;
    }
    return;
  }
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  const LagRanges3 R = lag_ranges3(a, g);
  PeakAcc acc;
  acc.best = 0.0;
  acc.bidx = -1;
  acc.smax = -INFINITY;
  acc.ssum = 0.0;
  for (int q = q0 + threadIdx.x; q < q1; q += K3C_THREADS) k3c_pair<N, ALG>(a, g, s, ci, q, P1, P2, P3, R, acc);
  // block merge: (largest value, lowest column-major index), NaN-propagating max, sum
  __shared__ double rb[K3C_THREADS / 32], rs[K3C_THREADS / 32], rm[K3C_THREADS / 32];
  __shared__ int ri[K3C_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double best = acc.best;
  int bidx = acc.bidx;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, off);
    const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
    peak_merge(best, bidx, ob, oi);
  }
  const double smax = warp_nmax3(acc.smax);
  const double ssum = warp_sum3(acc.ssum);
  if (lane == 0) {
    rb[warp] = best;
    ri[warp] = bidx;
    rm[warp] = smax;
    rs[warp] = ssum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = rb[0], mx = rm[0], sum = rs[0];
    int bi = ri[0];
    for (int w = 1; w < K3C_THREADS / 32; ++w) {
      peak_merge(b, bi, rb[w], ri[w]);
      mx = nmax(mx, rm[w]);
      sum += rs[w];
    }
    PeakPart3 pp;
    pp.best = b;
    pp.smax = mx;
    pp.ssum = sum;
    pp.bidx = bi;
    pp.pad_ = 0;
    a.cpart[ci * gridDim.x + part] = pp;
  }
}

// One thread per IA: its K3c parts in part order, then the Gaussian fit and
// SN from the similarity volume (k3c_final).
template <int N, int ALG>
__global__ void k3c_merge_kernel(Piv3dArgs a, long long n, int parts) {
  const long long ci = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= n) return;
  if (a.state[ci].skip) {
    k3c_skipped(a, ci);
    return;
  }
  const PeakPart3* p = a.cpart + ci * parts;
  double b = p[0].best, mx = p[0].smax, sum = p[0].ssum;
  int bi = p[0].bidx;
  for (int k = 1; k < parts; ++k) {
    peak_merge(b, bi, p[k].best, p[k].bidx);
    mx = nmax(mx, p[k].smax);
    sum += p[k].ssum;
  }
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  k3c_final(a, g, ci, lag_ranges3(a, g), b, bi, mx, sum);
}

// Last lags whose sums the pass's map holds.
__device__ __forceinline__ void mapped_lags3(const Piv3dArgs& a, const IAGeom3& g, const LagRanges3& R, int (&e)[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int size = d == 0 ? a.H : (d == 1 ? a.W : a.D);
    e[d] = min(R.hi[d], lag_mapped_max(a.SM[d], a.IS[d], g.g0[d], g.hi[d], size));
  }
}

// The walk's value of one lag (k3c_walk_kernel's) from its raw correlation; a
// lag that the map does not hold: +inf.
template <int ALG>
__device__ __forceinline__ float walk_value3(const Piv3dArgs& a, const IAGeom3& g, const IA3State& st, const int (&e)[3],
                                             int s1, int s2, int s3, float sqF, float fscale, float c) {
  if (s1 > e[0] || s2 > e[1] || s3 > e[2]) return INFINITY;
  const long long w = (g.g0[0] + s1 + a.SM[0]) +
                      (long long)a.ldw1 * ((g.g0[1] + s2 + a.SM[1]) + (long long)a.ldw2 * (g.g0[2] + s3 + a.SM[2]));
  if (ALG == ALG_NSQECC) {
    const float2 m = __ldg(a.ws + w);
    int open = 0;
    return nsqecc_walk(m.x, m.y, c, -2.f * fscale, (float)st.sumF2, sqF, open);
  }
  int r0, r1, c0, c1, z0, z1;
  lag_window(s1, a.IS[0], g.g0[0], g.lo[0], g.hi[0], r0, r1);
  lag_window(s2, a.IS[1], g.g0[1], g.lo[1], g.hi[1], c0, c1);
  lag_window(s3, a.IS[2], g.g0[2], g.lo[2], g.hi[2], z0, z1);
  const double n = (double)(r1 - r0) * (double)(c1 - c0) * (double)(z1 - z0);
  const double2 m = __ldg(a.wz + w);
  const double SG = m.x - 2.0 * st.meanG * m.y + n * st.meanG * st.meanG;
  return c * fscale * rsqrtf((float)(SG > 0.0 ? SG : 0.0));
}

// K3c of a pass that ends in the walk (finish3_fast): the lag pair's inverse
// along k3, the raw correlations to V (the fit's neighbourhood), FP32
// approximations of the similarity to the block's two largest.  With the
// window sums in one 8-byte read per lag (ZNCC: 16) instead of eight FP64 ones
// (sixteen), no FP64 square roots, quotients or compares and 128 registers
// instead of 224..237, two blocks run on an SM.
template <int N, int ALG>
__global__ void __launch_bounds__(K3C_THREADS, N <= 64 ? 2 : 1) k3c_walk_kernel(Piv3dArgs a) {
  constexpr int M = N / 2, K3 = M + 1;
  const int part = blockIdx.x, parts = gridDim.x;
  const long long ci = blockIdx.y;
  const int P1 = 2 * a.SM[0] + 1, P2 = 2 * a.SM[1] + 1, P3 = 2 * a.SM[2] + 1, P12 = P1 * P2;
  const int q0 = P12 * part / parts, q1 = P12 * (part + 1) / parts;
  const IA3State st = a.state[ci];
  if (st.skip) return;
  const IAGeom3 g = ia_geom3(a, a.ia_begin + ci);
  const LagRanges3 R = lag_ranges3(a, g);
  const float sqF = sqrtf((float)st.sumF2), F2 = (float)st.sumF2;
  const float fscale = (float)cc_scale3<N>(), m2 = -2.f * fscale;
  int e[3];
  mapped_lags3(a, g, R, e);
  TopTwo t;
  t.b1 = t.b2 = 0.f;
  t.idx = -1;
  int open = 0;
#pragma unroll 1
  for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
    const int s1 = q % P1, s2 = q / P1;
    float2 x[M];
    c2r_k3<N>(a.C + ci * K3 * P12 + q, P12, x);
    float* vdst = a.V + ci * P12 * P3 + q;
    const bool in = s1 >= R.lo[0] && s1 <= (ALG == ALG_FFTCC ? R.hi[0] : e[0]) && s2 >= R.lo[1] &&
                    s2 <= (ALG == ALG_FFTCC ? R.hi[1] : e[1]);
    const int last = ALG == ALG_FFTCC ? R.hi[2] : e[2];
    const long long w0 = (g.g0[0] + s1 + a.SM[0]) +
                         (long long)a.ldw1 * ((g.g0[1] + s2 + a.SM[1]) + (long long)a.ldw2 * (g.g0[2] + a.SM[2]));
    const long long wk = (long long)a.ldw1 * a.ldw2;
    double nrc = 0.0;
    if (ALG == ALG_ZNCC) {
      int r0, r1, c0, c1;
      lag_window(s1, a.IS[0], g.g0[0], g.lo[0], g.hi[0], r0, r1);
      lag_window(s2, a.IS[1], g.g0[1], g.lo[1], g.hi[1], c0, c1);
      nrc = (double)(r1 - r0) * (double)(c1 - c0);
    }
    constexpr int B = ALG == ALG_ZNCC ? 4 : 8;  // lags whose sums are read before any is used
#pragma unroll
    for (int b = 0; b < N; b += B) {
      if (b >= P3) continue;
      float2 m[B];
      double2 mz[B];
      if (ALG != ALG_FFTCC && in && last >= R.lo[2]) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const long long w = w0 + wk * min(max(b + k, R.lo[2]), last);
          if (ALG == ALG_NSQECC) m[k] = __ldg(a.ws + w);
          else mz[k] = __ldg(a.wz + w);
        }
      }
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int s3 = b + k;
        if (s3 < P3) {
          const float2 z = x[fpos<M>(s3 >> 1)];
          const float c = (s3 & 1) ? z.y : z.x;
          vdst[(long long)s3 * P12] = c;
          if (in && s3 >= R.lo[2] && s3 <= last) {
            const int idx = q + P12 * s3;
            if (ALG == ALG_FFTCC) {
              first_take(t, c, idx);
            } else if (ALG == ALG_NSQECC) {
              top_take(t, nsqecc_walk(m[k].x, m[k].y, c, m2, F2, sqF, open), idx);
            } else {
              int z0, z1;
              lag_window(s3, a.IS[2], g.g0[2], g.lo[2], g.hi[2], z0, z1);
              const double n = nrc * (double)(z1 - z0);
              const double SG = mz[k].x - 2.0 * st.meanG * mz[k].y + n * st.meanG * st.meanG;
              top_take(t, c * fscale * rsqrtf((float)(SG > 0.0 ? SG : 0.0)), idx);
            }
          }
        }
      }
    }
  }
  // lags whose sums the map does not hold, in full
  if (ALG != ALG_FFTCC && (e[0] < R.hi[0] || e[1] < R.hi[1] || e[2] < R.hi[2])) {
    __syncthreads();  // V of this part
#pragma unroll 1
    for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) {
      const int s1 = q % P1, s2 = q / P1;
      if (s1 < R.lo[0] || s1 > R.hi[0] || s2 < R.lo[1] || s2 > R.hi[1]) continue;
#pragma unroll 1
      for (int s3 = s1 <= e[0] && s2 <= e[1] ? max(e[2] + 1, R.lo[2]) : R.lo[2]; s3 <= R.hi[2]; ++s3) {
        const int idx = q + P12 * s3;
        const float v = (float)full_sim3<ALG>(a, g, st, s1, s2, s3, (double)a.V[ci * P12 * P3 + idx] * cc_scale3<N>());
        top_take(t, ALG == ALG_ZNCC ? v * sqF : v, idx);  // on the walk's scale
      }
    }
  }
  if (open < 0) top_open(t);
  // the block's two largest
  __shared__ TopPart3 red[K3C_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o1 = __shfl_xor_sync(0xffffffffu, t.b1, off), o2 = __shfl_xor_sync(0xffffffffu, t.b2, off);
    const int oi = __shfl_xor_sync(0xffffffffu, t.idx, off);
    top_merge(t, o1, o2, oi);
  }
  if (lane == 0) red[warp] = TopPart3{t.b1, t.b2, t.idx, 0};
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) top_merge(t, red[w].b1, red[w].b2, red[w].idx);
    reinterpret_cast<TopPart3*>(a.cpart)[ci * parts + part] = TopPart3{t.b1, t.b2, t.idx, 0};
  }
}

// A block per IA: the walk's parts, every lag in full where they leave more
// than one open, and the Gaussian fit with a lane per neighbour.
constexpr int K3F_THREADS = 512;  // at most
template <int N, int ALG>
__global__ void __launch_bounds__(K3F_THREADS) k3c_walk_merge_kernel(Piv3dArgs a, int parts) {
  const long long ci = blockIdx.x, ia = a.ia_begin + ci;
  const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const IA3State st = a.state[ci];
  if (st.skip) {
    if (tid == 0) k3c_skipped(a, ci);
    return;
  }
  const IAGeom3 g = ia_geom3(a, ia);
  const LagRanges3 R = lag_ranges3(a, g);
  const int P1 = 2 * a.SM[0] + 1, P2 = 2 * a.SM[1] + 1, P3 = 2 * a.SM[2] + 1, P12 = P1 * P2;
  const float* V = a.V + ci * P12 * P3;
  const double scale = cc_scale3<N>();
  const TopPart3* p = reinterpret_cast<const TopPart3*>(a.cpart) + ci * parts;
  TopTwo t;
  t.b1 = p[0].b1;
  t.b2 = p[0].b2;
  t.idx = p[0].idx;
  for (int k = 1; k < parts; ++k) top_merge(t, p[k].b1, p[k].b2, p[k].idx);
  int bidx = t.b1 > 0.f ? t.idx : -1;
  // an all-zero window has no value above 0; sums outside the normal FP32
  // range and near ties take the full search
  const bool zero = ALG != ALG_FFTCC && st.sumF2 == 0.0;
  const bool full = ALG != ALG_FFTCC && !zero &&
                    (!(st.sumF2 > 1e-30 && st.sumF2 < 1e30) || (t.b1 > 0.f && t.b2 >= t.b1 * (1.f - PEAK_GAP)));
  if (zero) bidx = -1;
  if (full) {
    double best = 0.0;
    bidx = -1;
    const int n1 = R.hi[0] - R.lo[0] + 1, n2 = R.hi[1] - R.lo[1] + 1, n3 = R.hi[2] - R.lo[2] + 1;
    const int total = n1 > 0 && n2 > 0 && n3 > 0 ? n1 * n2 * n3 : 0;
    // Within the bounds of the approximations only the lags that they put in the
    // gap are evaluated: the box is walked again, a batch of values in flight.
    // Nearly equal maxima are ordinary where an area holds noise on a bright
    // background, and one block with the whole box in full (33^3 lags of 64
    // bytes) held its pass up: 128^3 NSQECC, IS 32, SM 16, step 16, noise 1056 -> 738 us.
    const bool every = !(st.sumF2 > 1e-30 && st.sumF2 < 1e30) || !(t.b1 < INFINITY);
    const float th = t.b1 * (1.f - PEAK_GAP), sqF = sqrtf((float)st.sumF2);
    int e[3];
    mapped_lags3(a, g, R, e);
    // lag (s1, s2, s3) of this thread, every NT-th of the box
    const int d1 = NT % n1, d2 = (NT / n1) % n2, d3 = NT / (n1 * n2);
    int s1 = R.lo[0] + tid % n1, s2 = R.lo[1] + (tid / n1) % n2, s3 = R.lo[2] + tid / (n1 * n2);
    auto step = [&]() {
      s1 += d1;
      s2 += d2;
      s3 += d3;
      if (s1 > R.hi[0]) {
        s1 -= n1;
        ++s2;
      }
      if (s2 > R.hi[1]) {
        s2 -= n2;
        ++s3;
      }
    };
    constexpr int B = 4;
#pragma unroll 1
    for (int q0 = tid; q0 < total; q0 += B * NT) {
      int lag[B];  // those to evaluate, -1 = not
#pragma unroll
      for (int k = 0; k < B; ++k) {
        lag[k] = s3 <= R.hi[2] ? s1 + P1 * s2 + P12 * s3 : -1;
        if (!every && lag[k] >= 0 && !(walk_value3<ALG>(a, g, st, e, s1, s2, s3, sqF, (float)scale, V[lag[k]]) >= th)) lag[k] = -1;
        step();
      }
#pragma unroll
      for (int k = 0; k < B; ++k) {
        if (lag[k] < 0) continue;
        const int u3 = lag[k] / P12, u2 = (lag[k] - u3 * P12) / P1, u1 = lag[k] - u3 * P12 - u2 * P1;
        peak_take(full_sim3<ALG>(a, g, st, u1, u2, u3, (double)V[lag[k]] * scale), lag[k], best, bidx);
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
      peak_merge(best, bidx, ob, oi);
    }
    __shared__ double rb[K3F_THREADS / 32];
    __shared__ int ri[K3F_THREADS / 32];
    if (lane == 0) {
      rb[warp] = best;
      ri[warp] = bidx;
    }
    __syncthreads();
    best = rb[0];
    bidx = ri[0];
    for (int w = 1; w < NT / 32; ++w) peak_merge(best, bidx, rb[w], ri[w]);
  }
  if (warp != 0) return;
  double r[3] = {-1.0, -1.0, -1.0};  // no peak: 1-based (0, 0, 0), displacement -(SM+1)
  if (bidx >= 0) {
    const int pk[3] = {bidx % P1, (bidx / P1) % P2, bidx / P12};
    bool inside = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      r[d] = pk[d];
      inside = inside && (pk[d] + 1 > 1 + g.tlf[d]) && (pk[d] + 1 < 1 + 2 * a.SM[d] - g.brb[d]);
    }
    if (inside) {
      // lane = (i + 1) + 3 (j + 1) + 9 (k + 1); the similarity volume is FP32
      float v = 0.f;
      if (lane < 27) {
        const int s1 = pk[0] - 1 + lane % 3, s2 = pk[1] - 1 + (lane / 3) % 3, s3 = pk[2] - 1 + lane / 9;
        v = (float)full_sim3<ALG>(a, g, st, s1, s2, s3, (double)V[s1 + P1 * s2 + P12 * s3] * scale);
      }
      double mn = (double)__shfl_sync(0xffffffffu, v, 0);
#pragma unroll
      for (int k = 0; k < 27; ++k) mn = nmin(mn, (double)__shfl_sync(0xffffffffu, v, k));
      const double lg = lane < 27 ? log(1.0 + (double)v - mn) : 0.0;
      const int from[7] = {13, 12, 14, 10, 16, 4, 22};  // peak, then the neighbours along dims 1, 2, 3
      double l[7];
#pragma unroll
      for (int k = 0; k < 7; ++k) l[k] = __shfl_sync(0xffffffffu, lg, from[k]);
      refine3d_from_logs(pk, l, r);
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) a.VF[3 * ia + d] = r[d] - a.SM[d] + g.d[d];
  }
}

// Threads of a K3c walk block: the multiple of 32 that leaves the fewest idle
// in the last round over P12 lag pairs (289: 160 of 320 slots a round instead
// of 256 of 512), the larger of equal ones.
int walk_threads(int pairs) {
  int best = K3C_THREADS;
  auto slots = [&](int t) { return (pairs + t - 1) / t * t; };
  for (int t = K3C_THREADS - 32; t >= 96; t -= 32)
    if (slots(t) < slots(best)) best = t;
  return best;
}

template <int N, bool FPRUNE, int ALG, typename T>
cudaError_t run_chunks(Piv3dArgs a, long long chunk, cudaStream_t s, std::string& err) {
  using L = Lay3<N, FPRUNE>;
  constexpr bool CAN_SHARE = ALG == ALG_FFTCC || ALG == ALG_NSQECC;
  const bool shared = CAN_SHARE && a.Gs != nullptr;
  const size_t smem = (size_t)L::SMEM_F2 * sizeof(float2);
  auto k3b = k3b_kernel<N, FPRUNE, false>;
  if constexpr (CAN_SHARE) {
    if (shared) k3b = k3b_kernel<N, FPRUNE, true>;
  }
  cudaError_t e = allow_dyn_smem(k3b, smem);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return e;
  }
  const long long begin = a.ia_begin, end = a.ia_end, layer = (long long)a.vf[0] * a.vf[1];
  long long l0 = 0, l1 = 0;  // layers whose z-spectra are in Gs / Fs
  constexpr int NPASS = ALG == ALG_MASK_NSQECC ? 2 : 1;
  const int P12 = (2 * a.SM[0] + 1) * (2 * a.SM[1] + 1);
  for (long long c0 = begin; c0 < end;) {
    long long n = end - c0 < chunk ? end - c0 : chunk;
    // as many layers as the scratch holds
    if (shared) n = std::min(n, (c0 / layer + a.layers) * layer - c0);
    a.ia_begin = c0;
    a.ia_end = c0 + n;
    const unsigned merge_blocks = (unsigned)((n + 127) / 128);
    if constexpr (CAN_SHARE) {
      if (shared) {
        const long long f = c0 / layer, f1 = (c0 + n - 1) / layer + 1;
        if (f < l0 || f1 > l1) {
          l0 = f;
          l1 = f1;
          a.l0 = (int)l0;
          const int th = std::min(256, (a.H + 31) / 32 * 32);
          k3s_lines_kernel<N, FPRUNE, T><<<dim3((a.H + th - 1) / th, a.W, (unsigned)(2 * (l1 - l0))), th, 0, s>>>(a);
        }
        if (ALG == ALG_FFTCC && !(a.threshold >= 0.0)) {  // neither sumF2 nor a skip test
          if ((e = cudaMemsetAsync(a.state, 0, (size_t)n * sizeof(IA3State), s)) != cudaSuccess) {
            err = std::string("piv3d state: ") + cudaGetErrorString(e);
            return e;
          }
        } else {
          k3s_state_kernel<T, ALG><<<(unsigned)n, K3A_THREADS, 0, s>>>(a);
        }
      }
    }
    for (int pass = 0; pass < NPASS; ++pass) {
      if (!shared) {
        k3a_kernel<N, FPRUNE, ALG, T><<<dim3(k3a_parts(N), (unsigned)n), K3A_THREADS, 0, s>>>(a, pass);
        if (pass == 0) k3a_merge_kernel<N, ALG><<<merge_blocks, 128, 0, s>>>(a, n);
      }
      k3b<<<dim3(L::K3, (unsigned)n), 2 * N, smem, s>>>(a, pass == 0 ? a.C : a.C2);
    }
    const int cparts = k3c_parts(N, P12);
    bool done = false;
    if constexpr (ALG != ALG_MASK_NSQECC) {
      // without a map (batch plans) the full K3c is the faster one
      if (finish3_fast(a, ALG) && (ALG == ALG_FFTCC || (ALG == ALG_ZNCC ? a.wz != nullptr : a.ws != nullptr))) {
        const int th = walk_threads((P12 + cparts - 1) / cparts);
        k3c_walk_kernel<N, ALG><<<dim3(cparts, (unsigned)n), th, 0, s>>>(a);
        // few areas: more threads each, for the boxes walked again (96^3 of 125 areas, all near ties: 597 us with
        // 128 threads, 471 with 512); many: 160^3, two passes, 2530 us with 128, 2570 with 512
        const int ft = ALG != ALG_FFTCC && n <= 1024 ? K3F_THREADS : 128;
        k3c_walk_merge_kernel<N, ALG><<<(unsigned)n, ft, 0, s>>>(a, cparts);
        done = true;
      }
    }
    if (!done) {
      k3c_kernel<N, ALG><<<dim3(cparts, (unsigned)n), K3C_THREADS, 0, s>>>(a);
      k3c_merge_kernel<N, ALG><<<merge_blocks, 128, 0, s>>>(a, n, cparts);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) {
      err = std::string("piv3d launch: ") + cudaGetErrorString(e);
      return e;
    }
    c0 += n;
  }
  return cudaSuccess;
}

template <int N, bool FPRUNE, typename T>
cudaError_t run_alg(const Piv3dArgs& a, int alg, long long chunk, cudaStream_t s, std::string& err) {
  switch (alg) {
    case ALG_FFTCC: return run_chunks<N, FPRUNE, ALG_FFTCC, T>(a, chunk, s, err);
    case ALG_ZNCC: return run_chunks<N, FPRUNE, ALG_ZNCC, T>(a, chunk, s, err);
    case ALG_NSQECC: return run_chunks<N, FPRUNE, ALG_NSQECC, T>(a, chunk, s, err);
    case ALG_MASK_NSQECC: return run_chunks<N, FPRUNE, ALG_MASK_NSQECC, T>(a, chunk, s, err);
    default: err = "unknown correlation algorithm"; return cudaErrorInvalidValue;
  }
}

template <int N, bool FPRUNE>
cudaError_t run_dt(const Piv3dArgs& a, int alg, long long chunk, cudaStream_t s, std::string& err) {
  return a.dtype == 0 ? run_alg<N, FPRUNE, float>(a, alg, chunk, s, err)
                      : run_alg<N, FPRUNE, double>(a, alg, chunk, s, err);
}

}  // namespace

int piv3d_fft_len(const int SS[3]) {
  int m = SS[0];
  if (SS[1] > m) m = SS[1];
  if (SS[2] > m) m = SS[2];
  if (m <= 32) return 32;
  if (m <= 64) return 64;
  if (m <= 128) return 128;  // only with every interSize <= 64 (launch_piv3d)
  return 0;
}

static bool piv3d_prune(const int IS[3], int N) { return IS[0] <= N / 2 && IS[1] <= N / 2 && IS[2] <= N / 2; }

// Chunk scratch of c IAs: Gz | Fz | C | C2 | V | state | K3a parts | K3c
// parts, each array 256-byte aligned.
namespace {
struct Scr3 {
  size_t b[8];
};
Scr3 scr3(const int IS[3], const int SM[3], int alg, size_t c, bool shared) {
  Scr3 r{};
  const int SS[3] = {IS[0] + 2 * SM[0], IS[1] + 2 * SM[1], IS[2] + 2 * SM[2]};
  const int N = piv3d_fft_len(SS);
  if (N == 0) return r;
  const size_t K3 = N / 2 + 1;
  const size_t NF = piv3d_prune(IS, N) ? N / 2 : N;
  const size_t P12 = (size_t)(2 * SM[0] + 1) * (2 * SM[1] + 1);
  const size_t P3 = 2 * SM[2] + 1;
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  r.b[0] = shared ? 0 : al(c * K3 * N * N * sizeof(float2));                  // Gz
  r.b[1] = shared ? 0 : al(c * K3 * NF * NF * sizeof(float2));                // Fz
  r.b[2] = al(c * K3 * P12 * sizeof(float2));                                 // C
  r.b[3] = alg == ALG_MASK_NSQECC ? r.b[2] : 0;                               // C2
  r.b[4] = al(c * P12 * P3 * sizeof(float));                                  // V
  r.b[5] = al(c * sizeof(IA3State));                                          // state
  r.b[6] = al(c * k3a_parts(N) * sizeof(ReducePart3));                        // K3a parts
  r.b[7] = al(c * (size_t)k3c_parts(N, (int)P12) * sizeof(PeakPart3));        // K3c parts
  return r;
}
}  // namespace

size_t piv3d_scratch_bytes(const int IS[3], const int SM[3], int alg, long long chunk, bool shared) {
  const Scr3 r = scr3(IS, SM, alg, (size_t)chunk, shared);
  size_t t = 0;
  for (size_t x : r.b) t += x;
  return t;
}

size_t piv3d_scratch_bytes_per_ia(const int IS[3], const int SM[3], int alg, bool shared) {
  // one IA's share, with the alignment of the eight arrays
  return piv3d_scratch_bytes(IS, SM, alg, 1, shared);
}

// Shared z-spectra (k3s_lines_kernel) of one layer, G then F; column pitches
// are odd multiples of 128 bytes so that a window's columns spread over the
// cache's sets.
static long long shared3d_pitch(long long H) { return ((H + 15) / 16 | 1) * 16; }

size_t piv3d_shared_bytes(const int IS[3], const int SM[3], long long H, long long W) {
  const int SS[3] = {IS[0] + 2 * SM[0], IS[1] + 2 * SM[1], IS[2] + 2 * SM[2]};
  const long long K3 = piv3d_fft_len(SS) / 2 + 1;
  return (size_t)(2 * K3 * shared3d_pitch(H) * W) * sizeof(float2);
}

void piv3d_bind_shared(Piv3dArgs& a, int layers, char* base) {
  const int SS[3] = {a.IS[0] + 2 * a.SM[0], a.IS[1] + 2 * a.SM[1], a.IS[2] + 2 * a.SM[2]};
  a.pitch = shared3d_pitch(a.H);
  a.zplane = a.pitch * a.W;
  a.lstride = a.zplane * (piv3d_fft_len(SS) / 2 + 1);
  a.layers = layers;
  a.Gs = (float2*)base;
  a.Fs = a.Gs + a.lstride * layers;
}

void piv3d_bind_scratch(Piv3dArgs& a, int alg, long long chunk, char* base, bool shared) {
  const Scr3 r = scr3(a.IS, a.SM, alg, (size_t)chunk, shared);
  size_t o = 0;
  a.Gz = (float2*)(base + o);
  o += r.b[0];
  a.Fz = (float2*)(base + o);
  o += r.b[1];
  a.C = (float2*)(base + o);
  o += r.b[2];
  a.C2 = r.b[3] ? (float2*)(base + o) : nullptr;
  o += r.b[3];
  a.V = (float*)(base + o);
  o += r.b[4];
  a.state = (IA3State*)(base + o);
  o += r.b[5];
  a.apart = (ReducePart3*)(base + o);
  o += r.b[6];
  a.cpart = (PeakPart3*)(base + o);
}

// Window-sum maps of a 3D pass: a thread per (i, j) and ZMAP positions along k.
namespace {
constexpr int ZMAP = 4;
__device__ __forceinline__ void window_sums3(const double* __restrict__ II, int H, int W, int D, int IS3, int SM3, int r0,
                                             int r1, int c0, int c1, int k0, int n3, double (&S)[ZMAP]) {
#pragma unroll
  for (int t = 0; t < ZMAP; ++t) {
    const int k = k0 + t - SM3;
    const int z0 = k > 0 ? k : 0, z1 = k + IS3 < D ? k + IS3 : D;
    S[t] = k0 + t < n3 ? box_sum3(II, H, W, r0, r1, c0, c1, z0, z1) : 0.0;
  }
}
__global__ void __launch_bounds__(256) window_map3_kernel(Piv3dArgs a, float2* ws, double2* wz, int n3) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
  if (u >= a.ldw1) return;
  const int i = u - a.SM[0], j = v - a.SM[1];
  const int r0 = i > 0 ? i : 0, r1 = i + a.IS[0] < a.H ? i + a.IS[0] : a.H;
  const int c0 = j > 0 ? j : 0, c1 = j + a.IS[1] < a.W ? j + a.IS[1] : a.W;
  const int k0 = blockIdx.z * ZMAP;
  double S2[ZMAP], S1[ZMAP];
  window_sums3(a.IIg2, a.H, a.W, a.D, a.IS[2], a.SM[2], r0, r1, c0, c1, k0, n3, S2);
  if (wz) window_sums3(a.IIg, a.H, a.W, a.D, a.IS[2], a.SM[2], r0, r1, c0, c1, k0, n3, S1);
#pragma unroll
  for (int t = 0; t < ZMAP; ++t) {
    if (k0 + t < n3) {
      const long long at = u + (long long)a.ldw1 * (v + (long long)a.ldw2 * (k0 + t));
      if (wz) {
        wz[at] = make_double2(S2[t], S1[t]);
      } else {
        const float q = (float)S2[t];
        ws[at] = make_float2(q, sqrtf(q));
      }
    }
  }
}
}  // namespace

bool piv3d_takes_map(const Piv3dArgs& a, int alg) {
  if ((alg != ALG_NSQECC && alg != ALG_ZNCC) || !finish3_fast(a, alg)) return false;
  const int n1 = winmap_ld(a.H, a.IS[0], a.SM[0]), n2 = winmap_ld(a.W, a.IS[1], a.SM[1]),
            n3 = winmap_ld(a.D, a.IS[2], a.SM[2]);
  if (n2 > 65535 || (n3 + ZMAP - 1) / ZMAP > 65535) return false;  // the map kernel's grid
  // As in 2D (piv2d_takes_map); without a map the pass ends in the full K3c.
  // Whole passes without and with it, us, at 256x256x192 unless said otherwise:
  //   NSQECC, length 32 (IS 16, SM 8): 0.15 lags a position 392, 431; 0.37 lags 612, 571; 1.2 lags 1276, 939
  //           length 64 (IS 32, SM 16): 0.28 lags 655, 755; 1.1 lags 1282, 1101; 2.0 lags 1837, 1484
  //   ZNCC,   length 32: 0.15 lags 677, 770; 0.37 lags 875, 892; 1.2 lags 1555, 1242
  //           length 64: 0.28 lags 1034, 1123; 0.8 lags (IS 24, SM 12, 303x239x110) 1187, 1098; 1.1 lags 1748, 1546
  // Up to length 64 it takes more areas than SMs as well: of fewer, the full K3c
  // runs all at once.  NSQECC, length 64: 125 areas 1.1 lags (160^3) 468, 511; 4.9 lags
  // (96^3) 371, 401; 216 areas 1.9 lags (160^3) 694, 605; length 32: 64 areas 1.1 lags (64^3) 92, 98;
  // 216 areas 1.2 lags (96^3) 148, 139.  Length 128 (IS 48, SM 24), whose areas take
  // several blocks: 27 areas 3.5 lags (96^3) 854, 783.
  const int SS[3] = {a.IS[0] + 2 * a.SM[0], a.IS[1] + 2 * a.SM[1], a.IS[2] + 2 * a.SM[2]};
  const int N = piv3d_fft_len(SS);
  const double least = N == 64 ? 0.6 : 0.4, areas = (double)(a.ia_end - a.ia_begin);
  int dev = 0;
  if (N <= 64 && cudaGetDevice(&dev) == cudaSuccess && areas <= device_sm_count(dev)) return false;
  const double lags = areas * (2 * a.SM[0] + 1) * (2 * a.SM[1] + 1) * (2 * a.SM[2] + 1);
  return lags >= least * n1 * n2 * n3;
}

size_t window_map3_bytes(const Piv3dArgs& a, int alg) {
  const size_t n = (size_t)winmap_ld(a.H, a.IS[0], a.SM[0]) * (size_t)winmap_ld(a.W, a.IS[1], a.SM[1]) *
                   (size_t)winmap_ld(a.D, a.IS[2], a.SM[2]);
  return n * (alg == ALG_ZNCC ? sizeof(double2) : sizeof(float2));
}

cudaError_t launch_window_map3(Piv3dArgs& a, int alg, void* base, cudaStream_t s) {
  a.ldw1 = winmap_ld(a.H, a.IS[0], a.SM[0]);
  a.ldw2 = winmap_ld(a.W, a.IS[1], a.SM[1]);
  const int n3 = winmap_ld(a.D, a.IS[2], a.SM[2]);
  float2* ws = alg == ALG_ZNCC ? nullptr : (float2*)base;
  double2* wz = alg == ALG_ZNCC ? (double2*)base : nullptr;
  const int th = std::min(256, (a.ldw1 + 31) / 32 * 32);
  window_map3_kernel<<<dim3((a.ldw1 + th - 1) / th, a.ldw2, (n3 + ZMAP - 1) / ZMAP), th, 0, s>>>(a, ws, wz, n3);
  a.ws = ws;
  a.wz = wz;
  return cudaGetLastError();
}

cudaError_t launch_piv3d(const Piv3dArgs& a, int alg, long long chunk, cudaStream_t s, std::string& err) {
  const int SS[3] = {a.IS[0] + 2 * a.SM[0], a.IS[1] + 2 * a.SM[1], a.IS[2] + 2 * a.SM[2]};
  const int N = piv3d_fft_len(SS);
  if (!direct3d_ok(a.IS, a.SM) && (chunk < 1 || chunk > 65535)) {
    err = "3D chunk must be in [1, 65535]";
    return cudaErrorInvalidValue;
  }
  if (a.ia_end <= a.ia_begin) return cudaSuccess;
  if (direct3d_ok(a.IS, a.SM)) return launch_piv3d_direct(a, alg, s, err);  // small windows: no chunk scratch
  const bool prune = piv3d_prune(a.IS, N);
  if (N == 64) return prune ? run_dt<64, true>(a, alg, chunk, s, err) : run_dt<64, false>(a, alg, chunk, s, err);
  if (N == 32) return prune ? run_dt<32, true>(a, alg, chunk, s, err) : run_dt<32, false>(a, alg, chunk, s, err);
  // search windows 65..128 (the coarse passes of interSize-64 refinements):
  // the same kernels at length 128, for interrogation windows up to 64
  if (N == 128 && prune) return run_dt<128, true>(a, alg, chunk, s, err);
  err = "3D search window (interSize + 2 searchMargin) above 128, or above 64 with an interSize above 64, is not supported";
  return cudaErrorInvalidValue;
}

}  // namespace mqp
