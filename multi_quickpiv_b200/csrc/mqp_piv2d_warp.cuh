// The fused 2D warp kernels (see mqp_piv2d.cuh) and their launches, as
// templates; mqp_piv2d_w*.cu instantiate the single-pair kernels of one FFT
// length each, mqp_piv2d_b*.cu the work-queue kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <string>

#include "mqp_finish.cuh"
#include "mqp_internal.h"
#include "mqp_stage.cuh"

namespace mqp {

// ---------------------------------------------------------------------------
// warp reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double warp_nmax(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = nmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ void warp_peak(double& best, int& bidx) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, off);
    const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
    peak_merge(best, bidx, ob, oi);
  }
}

// ---------------------------------------------------------------------------
// the fused kernel
// ---------------------------------------------------------------------------
// One interrogation area, the whole per-IA body of PIV_CPU's loop, for one
// warp.  GH is the warp's shared-memory workspace (Layout2d, sized for this
// IA's lag plane), tw the (cos, sin)(2 pi j / N) table.  LW: ZNCC with an
// N/2 x N/2 interrogation window forms its window sums on chip (lw_rows /
// lw_cols) instead of reading integral images.  STG: this IA's search window
// was staged into GH by the TMA (mqp_stage.cuh) on mbar's phase `phase`, and
// the IA stages window ia_next (>= 0) as soon as its own G spectra are dead.
template <int N, bool FPRUNE, int ALG, typename T, bool LW = false, bool STG = false>
__device__ __forceinline__ void piv2d_ia(const Piv2dArgs& a, long long ia, float2* GH, const float2* tw, int lane,
                                         const CUtensorMap* tmap = nullptr, uint64_t* mbar = nullptr,
                                         unsigned* phase = nullptr, long long ia_next = -1) {
  using Lay = Layout2d<N, FPRUNE>;
  constexpr int M = N / 2;
  constexpr bool MASKED = ALG == ALG_MASK_NSQECC;
  static_assert(!LW || ((ALG == ALG_ZNCC || ALG == ALG_NSQECC) && FPRUNE), "on-chip window sums: ZNCC / NSQECC");
  static_assert(!STG || (!MASKED && sizeof(T) == 4), "staged windows: FP32, unmasked");
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1;
  // the plane follows the largest user of the G region: spectra, the window-sum table, the staged tile
  constexpr int F_OFF = STG ? (LW && Lay::F_OFF_LW > Lay::F_OFF_STG ? Lay::F_OFF_LW : Lay::F_OFF_STG)
                            : (LW ? Lay::F_OFF_LW : Lay::F_OFF);
  float2* FH = GH + F_OFF;
  // the next IA's window into the dead G spectra (every lane calls it)
  auto stage_next = [&]() {
    if (STG && ia_next >= 0 && *phase != STAGE_OFF) {
      stage_fence();
      __syncwarp();
      if (lane == 0) {
        const IAGeom gn = ia_geom(a, (int)(ia_next % a.vf1), (int)(ia_next / a.vf1));
        stage_issue<N>(tmap, reinterpret_cast<float*>(GH), mbar, stage_x0(gn.g01), gn.g02);
      }
    }
  };
  double* lw = LW ? reinterpret_cast<double*>(GH) : nullptr;
  double* plane = reinterpret_cast<double*>(FH);
  float* c1buf = MASKED ? reinterpret_cast<float*>(FH + Lay::region2_f2(P1, P2)) : nullptr;
  const double scale = cc_scale<N>();
  // lag rows [0, lane_rows) go one per lane; a short tail of rows
  // (2*SM1+1 just above 32) is computed by the whole warp, lanes over s2
  const int lane_rows = (P1 - 32 > 0 && P1 - 32 <= 4) ? 32 : P1;
  const int v1 = (int)(ia % a.vf1), v2 = (int)(ia / a.vf1);
  int d1, d2;
  ia_pred(a, v1, v2, d1, d2);
  const IAGeom g = ia_geom(a, v1, v2);
  IAScalars sc;
  sc.meanF = 0.0;
  sc.meanG = 0.0;
  if (ALG == ALG_ZNCC) {
    // copy_*_minus_mean! (src/utils/zncc_ops.jl:7-25): IA mean and the mean
    // of the whole clipped search region
    sc.meanF = box_sum(a.II1, a.H, g.ir1, g.ir1 + a.IS1, g.ir2, g.ir2 + a.IS2) / ((double)a.IS1 * a.IS2);
    const double nG = (double)(g.hi1 - g.lo1) * (double)(g.hi2 - g.lo2);
    sc.meanG = box_sum(a.IIg, a.H, g.g01 + g.lo1, g.g01 + g.hi1, g.g02 + g.lo2, g.g02 + g.hi2) / nG;
  }
  const long long vfo = (long long)v1 + (long long)a.vf1 * v2;
  bool skipped = false;

  // One pass correlates one pair of inputs; masked NSQECC needs two
  // ((F*mask) with G, mask with G^2, mask_nsqecc.jl:151-155).
  constexpr int NPASS = MASKED ? 2 : 1;
#pragma unroll 1
  for (int pass = 0; pass < NPASS; ++pass) {
    const int pmode = MASKED ? (pass == 0 ? PASS_MASKED : PASS_MASK_SQ) : PASS_PLAIN;

    // ---- phase 1: F rows and G rows, r2c along dim 2 (one rolled body) ----
    // The loads of the next row are in flight while the current row is
    // transformed.
    constexpr int NJF = (Lay::NF + 31) / 32, NJ = NJF + N / 32;
    double vmax = -INFINITY, mmax = -INFINITY, sumsq = 0.0;
    if (STG) {
      // F rows from global memory (row_process reads them itself) while the
      // staged window lands; then every lane reads its G rows from the tile
      // before any lane writes spectra over it
#pragma unroll 1
      for (int job = 0; job < NJF; ++job) {
        const RowJob jf = row_job<N, FPRUNE>(a, g, lane, job);
        float none[N];
#pragma unroll
        for (int x = 0; x < N; ++x) none[x] = 0.f;
        if (jf.row < Lay::NF) row_process<N, FPRUNE, T, ALG == ALG_ZNCC>(a, sc, pmode, jf, none, GH, FH, vmax, mmax, sumsq);
      }
      // a copy that never lands (bounded wait) raises the status flag and
      // turns staging off for this warp: its rows come from global memory
      const bool armed = *phase != STAGE_OFF;
      const bool tiled = __all_sync(0xffffffffu, armed && stage_wait(mbar, *phase));  // one verdict per warp
      if (armed) {
        if (tiled) {
          *phase ^= 1u;
        } else {
          *phase = STAGE_OFF;
          if (a.status && lane == 0) atomicExch(a.status, 1);
        }
      }
      const float* tile = reinterpret_cast<const float*>(GH) + (g.g01 - stage_x0(g.g01));
      float gv[N / 32][N];
      RowJob jg[N / 32];
#pragma unroll
      for (int h = 0; h < N / 32; ++h) {
        jg[h] = row_job<N, FPRUNE>(a, g, lane, NJF + h);
        if (tiled) {
          const float* rowp = tile + jg[h].row;
#pragma unroll
          for (int x = 0; x < N; ++x)
            gv[h][x] = (jg[h].live && x >= jg[h].xlo && x < jg[h].xhi) ? rowp[x * StageTile<N>::ROWS] : 0.f;
        } else {
          row_load<N, T>(a, jg[h], gv[h]);
        }
      }
      __syncwarp();
      // unrolled: a runtime row index would put gv in local memory
#pragma unroll
      for (int h = 0; h < N / 32; ++h)
        row_process<N, FPRUNE, T, ALG == ALG_ZNCC>(a, sc, pmode, jg[h], gv[h], GH, FH, vmax, mmax, sumsq);
    } else {
    float buf[N];
    RowJob jn = row_job<N, FPRUNE>(a, g, lane, 0);
    row_load<N, T>(a, jn, buf);
#pragma unroll 1
    for (int job = 0; job < NJ; ++job) {
      const RowJob jc = jn;
      float cur[N];
#pragma unroll
      for (int x = 0; x < N; ++x) cur[x] = buf[x];
      if (job + 1 < NJ) {
        jn = row_job<N, FPRUNE>(a, g, lane, job + 1);
        row_load<N, T>(a, jn, buf);
      }
      if (!(jc.isF && jc.row >= Lay::NF))
        row_process<N, FPRUNE, T, ALG == ALG_ZNCC>(a, sc, pmode, jc, cur, GH, FH, vmax, mmax, sumsq);
    }
    }
    if (pass == 0) {
      vmax = warp_max(vmax);
      sc.sumF2 = warp_sum(sumsq);
      // skip_inter_region (src/utils/piv_ops.jl:134-157): the vector stays zero
      bool skip;
      if (MASKED) {
        mmax = warp_max(mmax);
        skip = (a.threshold > 0.0 && vmax < a.threshold) || (a.mask_threshold > 0.0 && mmax < a.mask_threshold);
      } else {
        skip = a.threshold >= 0.0 && vmax < a.threshold;
      }
      if (skip) {
        skipped = true;
        break;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int n = lane; n < M; n += 32) split_G_pair<N, FPRUNE>(GH, tw, n);
    __syncwarp();

    // ---- phases 2 and 3: one rolled loop of stages around one FFT body ----
    // The plane is row-contiguous: element (s1, s2) at s1*P2 + s2.
    {
      constexpr int RU = (M + 31) / 32;  // spectrum rows per lane
      const int NS2 = 6 * RU;            // phase-2 stages
      const int RL = (lane_rows + 31) / 32;
      float2 t[M];  // carried from the F stage (the product) into the I stage
#pragma unroll 1
      for (int job = 0; job < NS2 + RL; ++job) {
        if (job == NS2) __syncwarp();  // all spectra rows finished before phase 3
        bool active;
        int st = 0, h = 0, u = 0, s1 = 0;
        if (job < NS2) {
          const int q = job % 6;
          u = lane + 32 * (job / 6);
          h = q / 3;
          st = q % 3;
          active = u < M;
          if (active) stage_pre<N, FPRUNE>(st, h, GH + u * Lay::GSTR, FH + u * Lay::FSTR, t);
        } else {
          s1 = lane + 32 * (job - NS2);
          active = s1 < lane_rows;
          if (active) c2r_pre<N, FPRUNE>(s1, GH, t);
        }
        if (!active) continue;
        fft_reg<M, false>(t);
        if (job < NS2) {
          stage_post<N, FPRUNE>(st, h, u == 0, P1, GH + u * Lay::GSTR, t);
        } else {
          double* prow = plane + s1 * P2;
#pragma unroll
          for (int n = 0; n < M; ++n) {
            const float2 z = cconj(t[fpos<M>(n)]);
            if (2 * n < P2) prow[2 * n] = (double)z.x * scale;
            if (2 * n + 1 < P2) prow[2 * n + 1] = (double)z.y * scale;
          }
        }
      }
    }
    __syncwarp();
    // raw correlation of the tail lag rows, all lanes over s2
#pragma unroll 1
    for (int s1 = lane_rows; s1 < P1; ++s1)
      for (int s2 = lane; s2 < P2; s2 += 32)
        plane[s1 * P2 + s2] = (double)tail_row_value<N, FPRUNE>(GH, tw, s1, s2) * scale;
    __syncwarp();
    if (!LW) stage_next();  // with LW the table holds the G region until the finish has read it
    if (LW) {
      // the G spectra are dead: their space takes the window-sum table
      lw_rows<N, T, ALG == ALG_ZNCC>(a, g, sc.meanG, lane, P2, lw);
      __syncwarp();
      lw_cols<N>(lane, P1, P2, lw);
      lw_col32<N>(lane, P1, P2, lw);
      __syncwarp();
    }
    if (MASKED && pass == 0) {
      // park (F*mask)*G while the second pass reuses the workspace
      for (int i = lane; i < P1 * P2; i += 32) c1buf[i] = (float)plane[i];
      __syncwarp();
    }
  }
  if (skipped) {
    stage_next();
    if (lane == 0) {
      a.VF[2 * vfo + 0] = 0.0;
      a.VF[2 * vfo + 1] = 0.0;
      if (a.SN) a.SN[vfo] = 0.0;
    }
    if (a.planes) {
      double* dst = a.planes + (ia - a.ia_begin) * (long long)P1 * P2;
      for (int i = lane; i < P1 * P2; i += 32) dst[i] = 0.0;
    }
    __syncwarp();
    return;
  }

  // ---- finish: similarity, peak (first_fullovp_peak), SN, Gaussian fit ----
  LagRanges R;
  R.lo1 = g.tlf1;
  R.hi1 = 2 * a.SM1 - g.brb1;
  R.lo2 = g.tlf2;
  R.hi2 = 2 * a.SM2 - g.brb2;
  R.shi1 = 2 * a.SM1 - 1 - g.brb1;
  R.shi2 = 2 * a.SM2 - 1 - g.brb2;
  if constexpr (MASKED) {
    if (finish_fast(a)) {
      auto c1 = [&](int s1, int s2) { return (double)c1buf[s1 * P2 + s2]; };
      auto c2 = [&](int s1, int s2) { return plane[s1 * P2 + s2]; };
      const int bidx = finish_search_masked<32>(a, g, sc, R, lane, P1, c1, c2, nullptr);
      double r1 = -1.0, r2 = -1.0;  // no peak: 1-based (0, 0), displacement -(SM+1)
      if (bidx >= 0)
        finish_refine_with(
            a, g, bidx % P1, bidx / P1, lane,
            [&](int s1, int s2) { return finish_one<ALG>(a, g, sc, s1, s2, c2(s1, s2), c1(s1, s2)); }, r1, r2);
      if (lane == 0) {
        a.VF[2 * vfo + 0] = r1 - a.SM1 + d1;
        a.VF[2 * vfo + 1] = r2 - a.SM2 + d2;
      }
      __syncwarp();
      return;
    }
  }
  if constexpr (!MASKED) {
    if (finish_fast(a)) {
      // the transforms' FP32 value: the plane's, times a power of two, may lie below FP32's normal range
      auto cc = [&](int s1, int s2) { return (float)(plane[s1 * P2 + s2] * (1.0 / cc_scale<N>())); };
      const int bidx = finish_search<ALG, 32, LW ? N : 0>(a, g, sc, R, lane, P1, scale, cc, lw, nullptr);
      double r1 = -1.0, r2 = -1.0;  // no peak: 1-based (0, 0), displacement -(SM+1)
      if (bidx >= 0)
        finish_refine<ALG, LW ? N : 0>(a, g, sc, bidx % P1, bidx / P1, lane, scale, cc, lw, r1, r2);
      __syncwarp();
      if (LW) stage_next();
      if (lane == 0) {
        a.VF[2 * vfo + 0] = r1 - a.SM1 + d1;
        a.VF[2 * vfo + 1] = r2 - a.SM2 + d2;
      }
      __syncwarp();
      return;
    }
  }
  PeakAcc acc;
  acc.best = 0.0;
  acc.bidx = -1;
  acc.smax = -INFINITY;
  acc.ssum = 0.0;
#pragma unroll 1
  for (int s1 = lane; s1 < lane_rows; s1 += 32)
    finish_row<ALG, LW ? N : 0>(a, g, sc, s1, P1, P2, plane + s1 * P2, R, acc, MASKED ? c1buf + s1 * P2 : nullptr,
                                lw);
#pragma unroll 1
  for (int s1 = lane_rows; s1 < P1; ++s1)
    for (int s2 = lane; s2 < P2; s2 += 32) {
      double& e = plane[s1 * P2 + s2];
      e = finish_one<ALG, LW ? N : 0>(a, g, sc, s1, s2, e, MASKED ? (double)c1buf[s1 * P2 + s2] : 0.0, lw);
      acc_take(acc, R, s1, s2, P1, e);
    }
  __syncwarp();
  if (LW) stage_next();
  double best = acc.best;
  int bidx = acc.bidx;
  warp_peak(best, bidx);
  double sn = 0.0;
  if (a.SN) {
    // compute_SN (src/utils/piv_ops.jl:336-367) over [TLF_off, 2SM-1-BRB_off]
    const double smax = warp_nmax(acc.smax);
    const double ssum = warp_sum(acc.ssum);
    const double len = (double)(R.shi1 - R.lo1 + 1) * (double)(R.shi2 - R.lo2 + 1);
    sn = smax / ((ssum - smax) / (len - 1.0));
  }
  if (a.planes) {
    double* dst = a.planes + (ia - a.ia_begin) * (long long)P1 * P2;
    for (int i = lane; i < P1 * P2; i += 32) dst[i] = plane[(i % P1) * P2 + i / P1];
  }
  double r1 = -1.0, r2 = -1.0;  // no peak: 1-based (0, 0), displacement -(SM+1)
  if (bidx >= 0) refine2d_warp(plane, P2, a.SM1, a.SM2, g, bidx % P1, bidx / P1, best, lane, r1, r2);
  if (lane == 0) {
    a.VF[2 * vfo + 0] = r1 - a.SM1 + d1;
    a.VF[2 * vfo + 1] = r2 - a.SM2 + d2;
    if (a.SN) a.SN[vfo] = sn;
  }
  __syncwarp();
}

// Persistent: each warp walks IAs ia = first + k * (all warps).  The warp's
// shared-memory workspace holds the spectra rows of G (N/2 x (N+1)) and F
// (N/2 x (NF+1)); after phase 2 the F rows are reused for the FP64 plane.
// STG: tmap describes img2 for the staged windows (mqp_stage.cuh); each
// warp stages its first window before the loop and every IA the next one.
template <int N, bool FPRUNE, int ALG, typename T, int WARPS, int MINB, bool LW = false, bool STG = false>
__global__ void __launch_bounds__(WARPS * 32, MINB) piv2d_kernel(Piv2dArgs a, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) float2 smem[];
  using Lay = Layout2d<N, FPRUNE>;
  constexpr bool MASKED = ALG == ALG_MASK_NSQECC;
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wf2 = STG ? Lay::warp_f2_stg(P1, P2) : (LW ? Lay::warp_f2_lw(P1, P2) : Lay::warp_f2(P1, P2, MASKED));
  float2* GH = smem + (size_t)warp * wf2;
  float2* tw = smem + (size_t)WARPS * wf2;  // (cos, sin)(2 pi j / N)
  uint64_t* mbar = reinterpret_cast<uint64_t*>(tw + N) + warp;
  for (int j = threadIdx.x; j < N; j += blockDim.x) tw[j] = twiddle_rt(j * (TW_N / N));
  if (STG && lane == 0) stage_init(mbar);
  __syncthreads();
  const long long nwarps = (long long)gridDim.x * WARPS;
  const long long first = a.ia_begin + (long long)blockIdx.x * WARPS + warp;
  unsigned phase = 0;
  if (STG && first < a.ia_end && lane == 0) {
    const IAGeom g0 = ia_geom(a, (int)(first % a.vf1), (int)(first / a.vf1));
    stage_issue<N>(&tmap, reinterpret_cast<float*>(GH), mbar, stage_x0(g0.g01), g0.g02);
  }
  for (long long ia = first; ia < a.ia_end; ia += nwarps)
    piv2d_ia<N, FPRUNE, ALG, T, LW, STG>(a, ia, GH, tw, lane, &tmap, mbar, &phase,
                                         ia + nwarps < a.ia_end ? ia + nwarps : -1);
}

// Batched: the IAs of many image pairs sharing one kernel variant form one
// work queue [0, total); prefix[k] is the first queue index of item k
// (prefix[n_items] = total).  Warps take `grab` consecutive queue entries at
// a time from `counter` (zeroed before the launch), so large and small pairs
// balance across the SMs.  wf2: float2 per warp, the largest any item needs.
template <int N, bool FPRUNE, int ALG, typename T, int WARPS, int MINB, bool LW = false>
__global__ void __launch_bounds__(WARPS * 32, MINB)
    piv2d_batch_kernel(const Piv2dArgs* __restrict__ items, const long long* __restrict__ prefix, int n_items,
                       long long total, int wf2, int grab, unsigned long long* counter) {
  extern __shared__ float2 smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* GH = smem + (size_t)warp * wf2;
  float2* tw = smem + (size_t)WARPS * wf2;
  for (int j = threadIdx.x; j < N; j += blockDim.x) tw[j] = twiddle_rt(j * (TW_N / N));
  __syncthreads();
  for (;;) {
    unsigned long long g0 = 0;
    if (lane == 0) g0 = atomicAdd(counter, (unsigned long long)grab);
    g0 = __shfl_sync(0xffffffffu, g0, 0);
    if ((long long)g0 >= total) break;
    for (int t = 0; t < grab; ++t) {
      const long long gi = (long long)g0 + t;
      if (gi >= total) break;
      int lo = 0, hi = n_items - 1;  // last k with prefix[k] <= gi
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= gi) lo = mid;
        else hi = mid - 1;
      }
      const Piv2dArgs& a = items[lo];
      piv2d_ia<N, FPRUNE, ALG, T, LW>(a, a.ia_begin + (gi - prefix[lo]), GH, tw, lane);
    }
  }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
template <int N, bool FPRUNE, int ALG, typename T, int WARPS, int MINB, bool LW = false, bool STG = false>
static cudaError_t launch_t(const Piv2dArgs& a, cudaStream_t s, std::string& err, const CUtensorMap* tm = nullptr) {
  using Lay = Layout2d<N, FPRUNE>;
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1;
  const int wf2 = STG ? Lay::warp_f2_stg(P1, P2) : (LW ? Lay::warp_f2_lw(P1, P2) : Lay::warp_f2(P1, P2, ALG == ALG_MASK_NSQECC));
  const size_t smem = ((size_t)WARPS * wf2 + N + (STG ? WARPS : 0)) * sizeof(float2);
  auto kern = piv2d_kernel<N, FPRUNE, ALG, T, WARPS, MINB, LW, STG>;
  CUtensorMap tmap;
  memset(&tmap, 0, sizeof(tmap));
  if (tm) tmap = *tm;
  cudaError_t e = allow_dyn_smem(kern, smem);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return e;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem);
  if (e != cudaSuccess || per_sm < 1) {
    err = "piv2d kernel does not fit on an SM (shared memory " + std::to_string(smem) + " B)";
    return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
  }
  const long long n_ia = a.ia_end - a.ia_begin;
  long long blocks = (long long)device_sm_count(dev) * per_sm;
  const long long need = (n_ia + WARPS - 1) / WARPS;
  if (blocks > need) blocks = need;
  if (blocks < 1) return cudaSuccess;
  kern<<<(unsigned)blocks, WARPS * 32, smem, s>>>(a, tmap);
  e = cudaGetLastError();
  if (e != cudaSuccess) err = std::string("piv2d launch: ") + cudaGetErrorString(e);
  return e;
}

// FP32 FFTCC / NSQECC / ZNCC with staged windows when img2 qualifies.
// Measured on B200 (2048^2 vortex, step 8, whole pass, results
// bit-identical): NSQECC interSize 32 2.41 -> 2.22 ms, 24 2.06 -> 1.85, 16
// 0.86 -> 0.82; FFTCC 32 1.42 -> 1.27, 24 1.32 -> 1.18, 16 0.65 -> 0.52;
// ZNCC 24 2.55 -> 2.49 (ZNCC with interSize N/2 goes through launch_lw).
template <int N, bool FPRUNE, int WARPS, int MINB>
static bool launch_stg(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err, cudaError_t& e) {
  if (a.dtype != 0 || !stage_enabled() || (alg != ALG_FFTCC && alg != ALG_NSQECC && alg != ALG_ZNCC)) return false;
  CUtensorMap tm;
  if (!stage_tensor_map(&tm, a.img2, a.H, a.W, N)) return false;
  e = alg == ALG_FFTCC  ? launch_t<N, FPRUNE, ALG_FFTCC, float, WARPS, MINB, false, true>(a, s, err, &tm)
      : alg == ALG_ZNCC ? launch_t<N, FPRUNE, ALG_ZNCC, float, WARPS, MINB, false, true>(a, s, err, &tm)
                        : launch_t<N, FPRUNE, ALG_NSQECC, float, WARPS, MINB, false, true>(a, s, err, &tm);
  return true;
}

template <int N, bool FPRUNE, typename T, int WARPS, int MINB>
static cudaError_t launch_alg(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err) {
  switch (alg) {
    case ALG_FFTCC: return launch_t<N, FPRUNE, ALG_FFTCC, T, WARPS, MINB>(a, s, err);
    case ALG_ZNCC: return launch_t<N, FPRUNE, ALG_ZNCC, T, WARPS, MINB>(a, s, err);
    case ALG_NSQECC: return launch_t<N, FPRUNE, ALG_NSQECC, T, WARPS, MINB>(a, s, err);
    // length 64: 29.7 KB per warp, three warps per block keep two blocks per SM
    case ALG_MASK_NSQECC: return launch_t<N, FPRUNE, ALG_MASK_NSQECC, T, N == 32 ? 4 : 3, MINB>(a, s, err);
    default: err = "unknown correlation algorithm"; return cudaErrorInvalidValue;
  }
}

template <int N, bool FPRUNE, int WARPS, int MINB>
static cudaError_t launch_dt(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err) {
  return a.dtype == 0 ? launch_alg<N, FPRUNE, float, WARPS, MINB>(a, alg, s, err)
                      : launch_alg<N, FPRUNE, double, WARPS, MINB>(a, alg, s, err);
}

template <int N, int MINB>
static cudaError_t launch_lw(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err) {
  if (alg != ALG_ZNCC) {
    err = "on-chip window sums are built for ZNCC";
    return cudaErrorInvalidValue;
  }
  // staged windows as well at length 32 (interSize 16: 0.98 -> 0.86 ms per 2048^2 pass); at length 64
  // the tile can only be issued after the finish has read the table, and the pass ran 2.77 -> 3.09 ms
  CUtensorMap tm;
  if (N == 32 && a.dtype == 0 && stage_enabled() && stage_tensor_map(&tm, a.img2, a.H, a.W, N))
    return launch_t<N, true, ALG_ZNCC, float, 4, MINB, true, true>(a, s, err, &tm);
  return a.dtype == 0 ? launch_t<N, true, ALG_ZNCC, float, 4, MINB, true>(a, s, err)
                      : launch_t<N, true, ALG_ZNCC, double, 4, MINB, true>(a, s, err);
}

template <int N, bool FPRUNE, int ALG, typename T, int WARPS, int MINB, bool LW = false>
static cudaError_t launch_batch_t(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  const size_t smem = ((size_t)WARPS * b.wf2 + N) * sizeof(float2);
  auto kern = piv2d_batch_kernel<N, FPRUNE, ALG, T, WARPS, MINB, LW>;
  cudaError_t e = allow_dyn_smem(kern, smem);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return e;
  }
  int dev = 0, per_sm = 0;
  cudaGetDevice(&dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem);
  if (e != cudaSuccess || per_sm < 1) {
    err = "piv2d batch kernel does not fit on an SM (shared memory " + std::to_string(smem) + " B)";
    return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
  }
  long long blocks = (long long)device_sm_count(dev) * per_sm;
  const long long need = (b.total + WARPS - 1) / WARPS;
  if (blocks > need) blocks = need;
  if (blocks < 1) return cudaSuccess;
  if ((e = cudaMemsetAsync(b.counter, 0, sizeof(unsigned long long), s)) != cudaSuccess) {
    err = std::string("counter reset: ") + cudaGetErrorString(e);
    return e;
  }
  kern<<<(unsigned)blocks, WARPS * 32, smem, s>>>(b.items, b.prefix, b.n_items, b.total, b.wf2,
                                                   b.grab > 0 ? b.grab : 1, b.counter);
  e = cudaGetLastError();
  if (e != cudaSuccess) err = std::string("piv2d batch launch: ") + cudaGetErrorString(e);
  return e;
}

template <int N, bool FPRUNE, typename T>
static cudaError_t launch_batch_alg(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  constexpr int MINB = N == 32 ? 3 : 2;  // as launch_piv2d
  switch (b.alg) {
    case ALG_FFTCC: return launch_batch_t<N, FPRUNE, ALG_FFTCC, T, 4, MINB>(b, s, err);
    case ALG_ZNCC: return launch_batch_t<N, FPRUNE, ALG_ZNCC, T, 4, MINB>(b, s, err);
    case ALG_NSQECC: return launch_batch_t<N, FPRUNE, ALG_NSQECC, T, 4, MINB>(b, s, err);
    case ALG_MASK_NSQECC: return launch_batch_t<N, FPRUNE, ALG_MASK_NSQECC, T, N == 32 ? 4 : 3, MINB>(b, s, err);
    default: err = "unknown correlation algorithm"; return cudaErrorInvalidValue;
  }
}

template <int N, int MINB>
static cudaError_t launch_batch_lw(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  if (b.alg != ALG_ZNCC) {
    err = "on-chip window sums are built for ZNCC";
    return cudaErrorInvalidValue;
  }
  return b.dtype == 0 ? launch_batch_t<N, true, ALG_ZNCC, float, 4, MINB, true>(b, s, err)
                      : launch_batch_t<N, true, ALG_ZNCC, double, 4, MINB, true>(b, s, err);
}

template <int N, bool FPRUNE>
static cudaError_t launch_batch_dt(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  return b.dtype == 0 ? launch_batch_alg<N, FPRUNE, float>(b, s, err) : launch_batch_alg<N, FPRUNE, double>(b, s, err);
}

}  // namespace mqp
