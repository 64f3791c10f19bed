// Peak search of the FFT kernels without the full similarity of every lag,
// and the window-sum maps it reads.
//
// A pass that returns no SN needs the similarity of few lags: the maximum's
// and its 3x3 neighbourhood's.  finish_search walks the lag box with FP32
// approximations of the similarity, keeps every lane's largest and
// second-largest value, and evaluates in full (finish_one: the values every
// other path forms) only what the approximation leaves open: one lag where
// the largest approximate value is alone within PEAK_GAP of the maximum, the
// whole box otherwise.  The result is the full search's: the approximations
// are within 1.5e-6 of the values they stand for (below), so a lag more than
// PEAK_GAP below the largest cannot be the maximum.
//
// NSQECC, v = d / (d + n) with d = sqrt(S2) sqrt(F2) and n = F2 + S2 - 2c
// (nsqecc_ops.jl:1-25): d is formed from the same FP32 square roots as in
// similarity_value.  n >= 0 up to the correlation's rounding (Cauchy), so
// F2 + S2 <= d + n + 4d and the terms of d + n add up to at most five times
// their sum; with three FP32 roundings each, the sum is within 9e-7 of exact,
// the approximate reciprocal and the product add 2e-7, and the full value's
// own FP32 steps 2e-7.  ZNCC, v = c / (sqrt(SG) sqrt(F2)) (zncc_ops.jl:29-50):
// SG is formed in FP64 as in similarity_value, its approximate inverse square
// root and the product are within 4e-7, the full value within 2e-7; the
// factor 1 / sqrt(F2) is common to the box and left out.
#pragma once

#include "mqp_piv2d.cuh"

namespace mqp {

constexpr float PEAK_GAP = 1e-5f;

// ---------------------------------------------------------------------------
// window-sum maps
// ---------------------------------------------------------------------------
// ws[(i + SM1) + ldw (j + SM2)] = (S2, sqrt(S2)) in FP32, S2 the FP64 sum of
// img2^2 over the interrogation-sized window at (i, j) clipped to the image
// (integral-image differences in box_sum's order), for i in [-SM1, H - IS1 +
// SM1] and j likewise: one 8-byte read per lag instead of four FP64 reads, and
// the square root once per window position instead of once per lag and IA.
MQP_HD MQP_FI int winmap_ld(int H, int IS, int SM) { return H - IS + 2 * SM + 1; }

// Last lag along an axis whose window sum is the map's: windows clip at the
// search region's end hi, which is the image's except in IAs that the border
// offset Q1 moves (their last lags' windows end short of the map's).
MQP_HD MQP_FI int lag_mapped_max(int SM, int IS, int g0, int hi, int size) {
  const int last = g0 + hi >= size ? 2 * SM : hi - IS;
  return last < 2 * SM ? last : 2 * SM;
}

// a lane's two largest values and the lag index of the largest
struct TopTwo {
  float b1, b2;
  int idx;
};
MQP_HD MQP_FI void top_take(TopTwo& t, float v, int idx) {
  if (v > t.b1) {
    t.b2 = t.b1;
    t.b1 = v;
    t.idx = idx;
  } else if (v > t.b2) {
    t.b2 = v;
  }
}

// exact values (FFTCC): the largest, and of equal ones the lowest index
MQP_HD MQP_FI void first_take(TopTwo& t, float v, int idx) {
  if (v > t.b1 || (v == t.b1 && idx < t.idx)) {
    t.b1 = v;
    t.idx = idx;
  }
}

#if defined(__CUDACC__)

__device__ __forceinline__ float rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.f / x;
#endif
}

// The lags of the box that the map does not hold (rows past e1, then columns
// past e2), over the lanes.
template <typename F>
__device__ __forceinline__ void unmapped_lags(const LagRanges& R, int e1, int e2, int lane, F take) {
  const int w2 = R.hi2 - R.lo2 + 1, nr = R.hi1 > e1 ? (R.hi1 - (e1 > R.lo1 - 1 ? e1 : R.lo1 - 1)) * w2 : 0;
  const int h1 = e1 - R.lo1 + 1, nc = R.hi2 > e2 && h1 > 0 ? (R.hi2 - (e2 > R.lo2 - 1 ? e2 : R.lo2 - 1)) * h1 : 0;
#pragma unroll 1
  for (int q = lane; q < nr + nc; q += 32) {
    if (q < nr) take(R.hi1 - q / w2, R.lo2 + q % w2);
    else take(R.lo1 + (q - nr) % h1, R.hi2 - (q - nr) / h1);
  }
}

// Lag box walk of one warp.  cc(s1, s2) is the raw correlation before the
// transforms' scale; rows s1 < lane_rows go one per lane (s1 = lane + 32 k),
// the others lanes over s2.  Returns the first maximum > 0 in column-major
// order (bidx = s1 + P1 s2, -1 = none), on every lane.
template <int ALG, typename CC>
__device__ __forceinline__ int finish_search(const Piv2dArgs& a, const IAGeom& g, const IAScalars& sc,
                                             const LagRanges& R, int lane, int lane_rows, int P1, double scale,
                                             CC cc) {
  const unsigned FULL = 0xffffffffu;
  const float sqF = sqrtf((float)sc.sumF2), F2 = (float)sc.sumF2;
  const float m2 = -2.f * (float)scale;
  TopTwo t;
  t.b1 = t.b2 = 0.f;
  t.idx = -1;
  bool full = false;  // every lag of the box in full
  if (ALG == ALG_FFTCC) {
    for (int s1 = lane; s1 < lane_rows; s1 += 32)
      if (s1 >= R.lo1 && s1 <= R.hi1) {
#pragma unroll 4
        for (int s2 = R.lo2; s2 <= R.hi2; ++s2) first_take(t, cc(s1, s2), s1 + P1 * s2);
      }
    for (int s1 = lane_rows > R.lo1 ? lane_rows : R.lo1; s1 <= R.hi1; ++s1)
      for (int s2 = R.lo2 + lane; s2 <= R.hi2; s2 += 32) first_take(t, cc(s1, s2), s1 + P1 * s2);
  } else {
    // outside this range the approximations could leave the normal FP32 range
    full = !(sc.sumF2 > 1e-30 && sc.sumF2 < 1e30);
    const int m1 = lag_mapped_max(a.SM1, a.IS1, g.g01, g.hi1, a.H), e1 = m1 < R.hi1 ? m1 : R.hi1;
    const int m2l = lag_mapped_max(a.SM2, a.IS2, g.g02, g.hi2, a.W), e2 = m2l < R.hi2 ? m2l : R.hi2;
    const float2* w0 = a.ws + (g.g01 + a.SM1) + (long long)a.ldw * (g.g02 + a.SM2);
    auto value = [&](float2 w, float c) {
      const float d = w.y * sqF;
      const float n = fmaf(m2, c, F2 + w.x);
      return d * rcp_approx(n + d);
    };
    if (!full) {
      for (int s1 = lane; s1 < lane_rows; s1 += 32)
        if (s1 >= R.lo1 && s1 <= e1) {
          for (int b = R.lo2; b <= e2; b += 8) {
            float2 q[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)  // past the box: its last column again, not taken
              q[k] = __ldg(w0 + s1 + (long long)a.ldw * min(b + k, e2));
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float v = value(q[k], cc(s1, min(b + k, e2)));
              if (b + k <= e2) top_take(t, v, s1 + P1 * (b + k));
            }
          }
        }
      for (int s1 = lane_rows > R.lo1 ? lane_rows : R.lo1; s1 <= e1; ++s1)
        for (int s2 = R.lo2 + lane; s2 <= e2; s2 += 32)
          top_take(t, value(__ldg(w0 + s1 + (long long)a.ldw * s2), cc(s1, s2)), s1 + P1 * s2);
      unmapped_lags(R, e1, e2, lane, [&](int s1, int s2) {
        top_take(t, (float)finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale), s1 + P1 * s2);
      });
    }
  }
  // the largest value of the box, and what comes within the gap of it
  float mx = t.b1;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, off));
  if (!full) {
    if (!(mx > 0.f)) return -1;
    if (ALG == ALG_FFTCC) {  // exact values: the first of equal maxima
      int idx = t.b1 == mx ? t.idx : 0x7fffffff;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) idx = min(idx, __shfl_xor_sync(FULL, idx, off));
      return idx;
    }
    const float th = mx * (1.f - PEAK_GAP);
    const unsigned near = __ballot_sync(FULL, t.b1 >= th);
    if (__popc(near) == 1 && !__any_sync(FULL, t.b2 >= th)) return __shfl_sync(FULL, t.idx, __ffs(near) - 1);
  }
  double best = 0.0;
  int bidx = -1;
  const int w2 = R.hi2 - R.lo2 + 1, total = (R.hi1 - R.lo1 + 1) * w2;
#pragma unroll 1
  for (int q = lane; q < total; q += 32) {
    const int s1 = R.lo1 + q / w2, s2 = R.lo2 + q % w2;
    peak_take(finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale), s1 + P1 * s2, best, bidx);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ob = __shfl_xor_sync(FULL, best, off);
    const int oi = __shfl_xor_sync(FULL, bidx, off);
    peak_merge(best, bidx, ob, oi);
  }
  return bidx;
}

// refine2d_warp from the raw correlations: nine lanes evaluate the 3x3
// neighbourhood of the peak (p1, p2) in full.
template <int ALG, typename CC>
__device__ __forceinline__ void finish_refine(const Piv2dArgs& a, const IAGeom& g, const IAScalars& sc, int p1, int p2,
                                              int lane, double scale, CC cc, double& r1, double& r2) {
  const unsigned FULL = 0xffffffffu;
  r1 = p1;
  r2 = p2;
  // refine2d_values' test
  const bool inside = (p1 + 1 > 1 + g.tlf1) && (p2 + 1 > 1 + g.tlf2) && (p1 + 1 < 1 + 2 * a.SM1 - g.brb1) &&
                      (p2 + 1 < 1 + 2 * a.SM2 - g.brb2);
  if (!inside) return;
  double v = 0.0;
  if (lane < 9) {
    const int s1 = p1 - 1 + lane % 3, s2 = p2 - 1 + lane / 3;
    v = finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale);
  }
  double mn = __shfl_sync(FULL, v, 0);
#pragma unroll
  for (int k = 0; k < 9; ++k) mn = nmin(mn, __shfl_sync(FULL, v, k));
  // the fit's five values sit on lanes 4 (peak), 3, 5 (along dim 1), 1, 7 (along dim 2)
  const double lg = lane < 9 ? log(1.0 + v - mn) : 0.0;
  const double l[5] = {__shfl_sync(FULL, lg, 4), __shfl_sync(FULL, lg, 3), __shfl_sync(FULL, lg, 5),
                       __shfl_sync(FULL, lg, 1), __shfl_sync(FULL, lg, 7)};
  refine2d_from_logs(p1, p2, l, r1, r2);
}

#endif  // __CUDACC__

}  // namespace mqp
