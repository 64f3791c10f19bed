// Peak search of the FFT kernels without the full similarity of every lag,
// and the window-sum maps it reads.
//
// A pass that returns no SN needs the similarity of few lags: the maximum's
// and its 3x3 neighbourhood's.  finish_search walks the lag box with FP32
// approximations of the similarity, keeps every lane's largest and
// second-largest value, and evaluates in full (finish_one: the values every
// other path forms) only what the approximation leaves open: one lag where
// the largest approximate value is alone within PEAK_GAP of the maximum, the
// few there are or the whole box otherwise (settle_peak).  The result is the full search's: the approximations
// are within 1.6e-6 of the values they stand for (below), so a lag more than
// PEAK_GAP below the largest cannot be the maximum.
//
// NSQECC, v = d / (d + n) with d = sqrt(S2) sqrt(F2) and n = F2 + S2 - 2c
// (nsqecc_ops.jl:1-25): d is formed from the same FP32 square roots as in
// similarity_value.  By Cauchy, d + n = F2 + S2 + d - 2c is at least (F2 + S2) / 2
// - but c is the FP32 transforms' correlation, whose error grows with the whole
// search window: beside pixels some 10^6 times brighter the sum may cancel.  A
// lag whose sum falls below a quarter of F2 + S2 sends the area to the full
// search (nsqecc_walk).  Above that the terms of the sum add up to at most
// seven times it; F2 and S2 in FP32 and the three FP32 additions leave it
// within 8e-7 of exact, the approximate reciprocal and the product add 2e-7,
// and the full value's own FP32 steps 2e-7.  ZNCC, v = c / (sqrt(SG) sqrt(F2))
// (zncc_ops.jl:29-50): SG is formed in FP64 as in similarity_value, its
// approximate inverse square root and the product are within 4e-7, the full
// value within 2e-7; the factor 1 / sqrt(F2) is common to the box and left out.
#pragma once

#include "mqp_piv2d.cuh"

namespace mqp {

constexpr float PEAK_GAP = 4e-6f;

// ---------------------------------------------------------------------------
// window-sum maps
// ---------------------------------------------------------------------------
// ws[(i + SM1) + ldw (j + SM2)] = (S2, sqrt(S2)) in FP32, S2 the FP64 sum of
// img2^2 over the interrogation-sized window at (i, j) clipped to the image
// (integral-image differences in box_sum's order), for i in [-SM1, H - IS1 +
// SM1] and j likewise: one 8-byte read per lag instead of four FP64 reads, and
// the square root once per window position instead of once per lag and IA.
// ZNCC: wz holds the FP64 sums of img2^2 and img2 (the variance about the search
// mean cancels), one 16-byte read instead of eight of 8 bytes.
MQP_HD MQP_FI int winmap_ld(int H, int IS, int SM) { return H - IS + 2 * SM + 1; }

// Last lag along an axis whose window sum is the map's: windows clip at the
// search region's end hi, which is the image's except in IAs that the border
// offset Q1 moves (their last lags' windows end short of the map's).
MQP_HD MQP_FI int lag_mapped_max(int SM, int IS, int g0, int hi, int size) {
  const int last = g0 + hi >= size ? 2 * SM : hi - IS;
  return last < 2 * SM ? last : 2 * SM;
}

// The lags of the box that the map does not hold: the rows past e1, then what
// the others have past column e2.
struct UnmappedLags {
  int w2, rows, h1, cols;  // lags of a row, lags in rows past e1, rows up to e1, lags past column e2
  MQP_HD MQP_FI int count() const { return rows + cols; }
  MQP_HD MQP_FI void at(const LagRanges& R, int q, int& s1, int& s2) const {
    s1 = q < rows ? R.hi1 - q / w2 : R.lo1 + (q - rows) % h1;
    s2 = q < rows ? R.lo2 + q % w2 : R.hi2 - (q - rows) / h1;
  }
};
MQP_HD MQP_FI UnmappedLags unmapped_lags(const LagRanges& R, int e1, int e2) {
  UnmappedLags u;
  u.w2 = R.hi2 - R.lo2 + 1;
  u.rows = R.hi1 > e1 ? (R.hi1 - (e1 > R.lo1 - 1 ? e1 : R.lo1 - 1)) * u.w2 : 0;
  u.h1 = e1 - R.lo1 + 1;
  u.cols = R.hi2 > e2 && u.h1 > 0 ? (R.hi2 - (e2 > R.lo2 - 1 ? e2 : R.lo2 - 1)) * u.h1 : 0;
  return u;
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

MQP_HD MQP_FI float rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.f / x;
#endif
}
MQP_HD MQP_FI float sqrt_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return sqrtf(x);
#endif
}
MQP_HD MQP_FI int sign_word(float x) {  // negative when x's sign bit is set
#if defined(__CUDA_ARCH__)
  return __float_as_int(x);
#else
  return signbit(x) ? -1 : 0;
#endif
}

// The walk's similarity of one lag from its raw correlation c; open turns
// negative (and stays so over the lags) where the approximation is not within
// the bounds above.  NSQECC: S2 and its root, m2 = -2 times the correlation's
// scale.
MQP_HD MQP_FI float nsqecc_walk(float S2, float root, float c, float m2, float F2, float sqF, int& open) {
  const float d = root * sqF, t = F2 + S2, den = fmaf(m2, c, t) + d;
  open |= sign_word(fmaf(-0.25f, t, den));
  return d * rcp_approx(den);
}
// Masked NSQECC, c1 = (F*mask)*G and S2 = mask*G^2; most keeps the largest
// magnitude, above 4 = open.
MQP_HD MQP_FI float masked_walk(double S2, double c1, double sumF2, float sqF, float& most) {
  const float d = sqrt_approx(fabsf((float)S2)) * sqF;
  const double n = ((sumF2 - 2.0 * c1) + S2) + (double)d;
  const float v = d * rcp_approx((float)n);
  most = fmaxf(most, fabsf(v));
  return v;
}
// A lane that met an open lag: two values no other lane's can exceed, so that
// the search does not end on one lag.
MQP_HD MQP_FI void top_open(TopTwo& t) { t.b1 = t.b2 = INFINITY; }

#if defined(__CUDACC__)

__device__ __forceinline__ float warp_most(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// The largest value of NT threads (barriers around red when NT > 32).
template <int NT>
__device__ __forceinline__ float block_most(int tid, float v, double* red) {
  v = warp_most(v);
  if (NT > 32) {
    float* rf = reinterpret_cast<float*>(red);
    if ((tid & 31) == 0) rf[tid >> 5] = v;
    __syncthreads();
    v = rf[0];
    for (int w = 1; w < NT / 32; ++w) v = fmaxf(v, rf[w]);
    __syncthreads();
  }
  return v;
}

// FFTCC, whose values are exact: the first of equal maxima above 0.
template <int NT>
__device__ __forceinline__ int first_of(int tid, const TopTwo& t, double* red) {
  const float mx = block_most<NT>(tid, t.b1, red);
  if (!(mx > 0.f)) return -1;
  int idx = t.b1 == mx ? t.idx : 0x7fffffff;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) idx = min(idx, __shfl_xor_sync(0xffffffffu, idx, off));
  if (NT > 32) {
    int* ri = reinterpret_cast<int*>(red);
    if ((tid & 31) == 0) ri[tid >> 5] = idx;
    __syncthreads();
    idx = ri[0];
    for (int w = 1; w < NT / 32; ++w) idx = min(idx, ri[w]);
    __syncthreads();
  }
  return idx;
}

// The peak from every thread's share t of the walk.  One lag alone within the
// gap of the largest is the peak.  Of several, each thread evaluates its own in
// full (sim); where a thread holds two, so that one's lag is not known, or
// full is set, all lags of the box are.  Nearly equal maxima are ordinary where
// an area holds noise on a bright background, and areas that take longer than
// their neighbours also cost the persistent kernels' warps their common pace
// through the code.  1024^2 passes, noise 100 wide on a background of 1000, whole
// box for any two in a gap of 1e-5 -> this with PEAK_GAP: NSQECC IS 16, SM 8 292 -> 204 us
// (every lag in full, no walk: 237), IS 12, SM 19 791 -> 415 (755), IS 32, SM 16 510 -> 408
// (571), masked IS 32 2506 -> 1661 (1632).
template <int NT, typename SIM>
__device__ __forceinline__ int settle_peak(const LagRanges& R, int tid, int P1, bool full, const TopTwo& t, double* red,
                                           SIM sim) {
  const unsigned FULL = 0xffffffffu;
  constexpr int NW = NT / 32;
  const int warp = tid >> 5, lane = tid & 31;
  float th = 0.f;
  if (!full) {
    const float mx = block_most<NT>(tid, t.b1, red);
    if (!(mx > 0.f)) return -1;
    th = mx * (1.f - PEAK_GAP);
    // threads with a value within the gap, above the 16th bit those with two, and the lag of an only one
    int cnt = (t.b1 >= th) + ((t.b2 >= th) << 16), idx = t.b1 >= th ? t.idx : -1;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      cnt += __shfl_xor_sync(FULL, cnt, off);
      idx = max(idx, __shfl_xor_sync(FULL, idx, off));
    }
    if (NT > 32) {
      int* ri = reinterpret_cast<int*>(red);
      if (lane == 0) {
        ri[2 * warp] = cnt;
        ri[2 * warp + 1] = idx;
      }
      __syncthreads();
      cnt = ri[0];
      idx = ri[1];
      for (int w = 1; w < NW; ++w) {
        cnt += ri[2 * w];
        idx = max(idx, ri[2 * w + 1]);
      }
      __syncthreads();
    }
    if (cnt == 1) return idx;
    full = cnt >> 16;
  }
  double best = 0.0;
  int bidx = -1;
  // this thread's lags: its one, or every NT-th of the box row by row
  const int w2 = R.hi2 - R.lo2 + 1, d1 = NT / w2, d2 = NT - d1 * w2;
  const int left = full ? ((R.hi1 - R.lo1 + 1) * w2 - tid + NT - 1) / NT : (t.b1 >= th);
  const int first = full ? tid / w2 : t.idx / P1, rest = full ? tid - first * w2 : t.idx - first * P1;
  int s1 = full ? R.lo1 + first : rest, s2 = full ? R.lo2 + rest : first;
#pragma unroll 1
  for (int k = 0; k < left; ++k) {
    peak_take(sim(s1, s2), s1 + P1 * s2, best, bidx);
    s1 += d1;
    s2 += d2;
    if (s2 > R.hi2) {
      s2 -= w2;
      ++s1;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ob = __shfl_xor_sync(FULL, best, off);
    const int oi = __shfl_xor_sync(FULL, bidx, off);
    peak_merge(best, bidx, ob, oi);
  }
  if (NT > 32) {
    if (lane == 0) {
      red[2 * warp] = best;
      red[2 * warp + 1] = (double)bidx;
    }
    __syncthreads();
    best = red[0];
    bidx = (int)red[1];
    for (int w = 1; w < NW; ++w) peak_merge(best, bidx, red[2 * w], (int)red[2 * w + 1]);
    __syncthreads();
  }
  return bidx;
}

// Lag box walk of NT threads (one warp, or a block whose every thread calls
// it).  cc(s1, s2) * scale is the raw correlation.  Returns the first maximum > 0
// in column-major order (bidx = s1 + P1 s2, -1 = none) on every thread.  Window
// sums come from the pass's map (a.ws, ZNCC: a.wz), from the on-chip table lw
// (LWN = N, mqp_piv2d.cuh) or, without either, from the integral images.  red:
// 2 NT / 32 doubles of shared memory when NT > 32 (the caller's barriers
// around it).
template <int ALG, int NT, int LWN, typename CC>
__device__ __forceinline__ int finish_search(const Piv2dArgs& a, const IAGeom& g, const IAScalars& sc,
                                             const LagRanges& R, int tid, int P1, double scale, CC cc,
                                             const double* lw, double* red) {
  static_assert(ALG == ALG_FFTCC || ALG == ALG_ZNCC || ALG == ALG_NSQECC, "unmasked similarities");
  const float sqF = sqrtf((float)sc.sumF2), F2 = (float)sc.sumF2;
  const float fscale = (float)scale, m2 = -2.f * fscale;
  TopTwo t;
  t.b1 = t.b2 = 0.f;
  t.idx = -1;
  // every lag of the box in full: also where the approximations could leave
  // the normal FP32 range
  const bool full = ALG != ALG_FFTCC && !(sc.sumF2 > 1e-30 && sc.sumF2 < 1e30);
  const bool map = ALG == ALG_NSQECC ? a.ws != nullptr : (ALG == ALG_ZNCC && !LWN && a.wz != nullptr);
  int e1 = R.hi1, e2 = R.hi2;
  if (map) {
    e1 = min(e1, lag_mapped_max(a.SM1, a.IS1, g.g01, g.hi1, a.H));
    e2 = min(e2, lag_mapped_max(a.SM2, a.IS2, g.g02, g.hi2, a.W));
  }
  // lag q of the walk: s1 = lo1 + q % w1, s2 = lo2 + q / w1, so that a warp
  // reads runs of consecutive rows
  const int w1 = e1 - R.lo1 + 1, total = w1 > 0 && e2 >= R.lo2 ? w1 * (e2 - R.lo2 + 1) : 0;
  int open = 0;
  if (!full && total > 0) {
    const int d2 = NT / w1, d1 = NT - d2 * w1;
    int s2 = R.lo2 + tid / w1, s1 = R.lo1 + tid % w1;
    auto step = [&]() {
      s1 += d1;
      s2 += d2;
      if (s1 > e1) {
        s1 -= w1;
        ++s2;
      }
    };
    if (ALG == ALG_FFTCC) {
#pragma unroll 4
      for (int q = tid; q < total; q += NT) {
        first_take(t, cc(s1, s2), s1 + P1 * s2);
        step();
      }
    } else {
      // B lags' correlations and sums (load) are read before any is used (value)
      auto walk = [&](auto load, auto value) {
        constexpr int B = 8;
        if (NT == 32 && w1 > 20) {
          // most of a warp's lanes find a row of their own: no index to keep per lag
          // (2048^2 NSQECC strips, step 8, rows and lags dealt out: 33 rows 1277, 1299 us; 17 rows
          // 1146, 1134; between them within 2 % of one another either way)
          const int s1 = min(R.lo1 + tid, e1);
          const bool mine = R.lo1 + tid <= e1;
#pragma unroll 1
          for (int b = R.lo2; b <= e2; b += B) {
            decltype(load(0, 0)) m[B];
#pragma unroll
            for (int k = 0; k < B; ++k) m[k] = load(s1, min(b + k, e2));
#pragma unroll
            for (int k = 0; k < B; ++k) {
              const float v = value(m[k], cc(s1, min(b + k, e2)));
              if (mine && b + k <= e2) top_take(t, v, s1 + P1 * (b + k));
            }
          }
#pragma unroll 1
          for (int u1 = R.lo1 + 32; u1 <= e1; ++u1)  // rows past the lanes, lanes over columns
            for (int u2 = R.lo2 + tid; u2 <= e2; u2 += 32) top_take(t, value(load(u1, u2), cc(u1, u2)), u1 + P1 * u2);
          return;
        }
#pragma unroll 1
        for (int q = tid; q < total; q += NT * B) {
          decltype(load(0, 0)) m[B];
          float c[B];
          int id[B];
#pragma unroll
          for (int k = 0; k < B; ++k) {
            const bool in = q + k * NT < total;
            id[k] = in ? s1 + P1 * s2 : -1;
            const int u1 = in ? s1 : R.lo1, u2 = in ? s2 : R.lo2;  // past the box: its first lag, not taken
            c[k] = cc(u1, u2);
            m[k] = load(u1, u2);
            step();
          }
#pragma unroll
          for (int k = 0; k < B; ++k) {
            const float v = value(m[k], c[k]);
            if (id[k] >= 0) top_take(t, v, id[k]);
          }
        }
      };
      auto nsqecc = [&](float s, float q, float c) { return nsqecc_walk(s, q, c, m2, F2, sqF, open); };
      auto zncc = [&](double S2, double S1, double n, float c) {
        const double SG = S2 - 2.0 * sc.meanG * S1 + n * sc.meanG * sc.meanG;
        return c * fscale * rsqrtf((float)(SG > 0.0 ? SG : 0.0));
      };
      const long long w0 = (g.g01 + a.SM1) + (long long)a.ldw * (g.g02 + a.SM2);
      auto window = [&](int u1, int u2, int& r0, int& r1, int& c0, int& c1) {
        lag_window(u1, a.IS1, g.g01, g.lo1, g.hi1, r0, r1);
        lag_window(u2, a.IS2, g.g02, g.lo2, g.hi2, c0, c1);
      };
      if (LWN) {
        walk([&](int u1, int u2) { return lw[lw_at(LWN, u1, u2)]; },
             [&](double S2, float c) { return c * fscale * rsqrtf((float)S2); });
      } else if (ALG == ALG_NSQECC && map) {
        const float2* w = a.ws + w0;
        walk([&](int u1, int u2) { return __ldg(w + (u1 + (long long)a.ldw * u2)); },
             [&](float2 m, float c) { return nsqecc(m.x, m.y, c); });
      } else if (ALG == ALG_NSQECC) {
        walk(
            [&](int u1, int u2) {
              int r0, r1, c0, c1;
              window(u1, u2, r0, r1, c0, c1);
              return box_sum(a.IIg2, a.H, r0, r1, c0, c1);
            },
            [&](double S2, float c) { return nsqecc((float)S2, sqrt_approx((float)S2), c); });
      } else if (map) {
        const double2* w = a.wz + w0;
        // interrogation-sized windows, but for those the image's edge cuts
        const double nw = (double)a.IS1 * (double)a.IS2;
        const bool whole = g.g01 + R.lo1 >= 0 && g.g01 + e1 + a.IS1 <= a.H && g.g02 + R.lo2 >= 0 && g.g02 + e2 + a.IS2 <= a.W;
        walk(
            [&](int u1, int u2) {
              const double2 v = __ldg(w + (u1 + (long long)a.ldw * u2));
              double n = nw;
              if (!whole) {
                int r0, r1, c0, c1;
                window(u1, u2, r0, r1, c0, c1);
                n = (double)(r1 - r0) * (double)(c1 - c0);
              }
              return make_double3(v.x, v.y, n);
            },
            [&](double3 m, float c) { return zncc(m.x, m.y, m.z, c); });
      } else {
        walk(
            [&](int u1, int u2) {
              int r0, r1, c0, c1;
              window(u1, u2, r0, r1, c0, c1);
              return make_double3(box_sum(a.IIg2, a.H, r0, r1, c0, c1), box_sum(a.IIg, a.H, r0, r1, c0, c1),
                                  (double)(r1 - r0) * (double)(c1 - c0));
            },
            [&](double3 m, float c) { return zncc(m.x, m.y, m.z, c); });
      }
    }
  }
  if (!full && map) {
    const UnmappedLags u = unmapped_lags(R, e1, e2);
#pragma unroll 1
    for (int q = tid; q < u.count(); q += NT) {
      int s1, s2;
      u.at(R, q, s1, s2);
      const float v = (float)finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale);
      top_take(t, ALG == ALG_ZNCC ? v * sqF : v, s1 + P1 * s2);  // on the walk's scale
    }
  }
  if (open < 0) top_open(t);
  if (ALG == ALG_FFTCC) return first_of<NT>(tid, t, red);
  return settle_peak<NT>(R, tid, P1, full, t, red, [&](int s1, int s2) {
    return finish_one<ALG, LWN>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale, 0.0, lw);
  });
}

// finish_search of masked NSQECC (masked_nsqecc_ops.jl:123-142): c1(s1, s2) is
// (F*mask)*G and c2 is mask*G^2, the window sum.  Both carry the FP32 transforms'
// error, so the denominator may cancel where the mask covers little: it is
// formed in FP64 as in similarity_value, and a value above 4 of either sign (a
// cancelled denominator, which scales the square root's approximation up and
// may come out of it with the other sign) takes the full search: up to there
// the root's 3e-7 leaves the value within 1.2e-6, its other steps add 4e-7.
template <int NT, typename C1, typename C2>
__device__ __forceinline__ int finish_search_masked(const Piv2dArgs& a, const IAGeom& g, const IAScalars& sc,
                                                    const LagRanges& R, int tid, int P1, C1 c1, C2 c2, double* red) {
  if (sc.sumF2 == 0.0) return -1;  // no lag has a value above 0
  const float sqF = sqrtf((float)sc.sumF2);
  const bool full = !(sc.sumF2 > 1e-30 && sc.sumF2 < 1e30);
  TopTwo t;
  t.b1 = t.b2 = 0.f;
  t.idx = -1;
  const int w1 = R.hi1 - R.lo1 + 1, w2 = R.hi2 - R.lo2 + 1, total = w1 > 0 && w2 > 0 ? w1 * w2 : 0;
  float most = 0.f;
  if (!full && total > 0) {
    const int d2 = NT / w1, d1 = NT - d2 * w1;
    int s2 = R.lo2 + tid / w1, s1 = R.lo1 + tid % w1;
#pragma unroll 4
    for (int q = tid; q < total; q += NT) {
      top_take(t, masked_walk(c2(s1, s2), c1(s1, s2), sc.sumF2, sqF, most), s1 + P1 * s2);
      s1 += d1;
      s2 += d2;
      if (s1 > R.hi1) {
        s1 -= w1;
        ++s2;
      }
    }
  }
  if (most > 4.f) top_open(t);
  return settle_peak<NT>(R, tid, P1, full, t, red, [&](int s1, int s2) {
    return finish_one<ALG_MASK_NSQECC>(a, g, sc, s1, s2, c2(s1, s2), c1(s1, s2));
  });
}

// Whether a pass ends in finish_search (masked: finish_search_masked).
MQP_HD MQP_FI bool finish_fast(const Piv2dArgs& a) { return a.SN == nullptr && a.planes == nullptr; }

// refine2d_warp from the raw correlations: nine lanes evaluate the 3x3
// neighbourhood of the peak (p1, p2) in full.
template <typename SIM>
__device__ __forceinline__ void finish_refine_with(const Piv2dArgs& a, const IAGeom& g, int p1, int p2, int lane,
                                                   SIM sim, double& r1, double& r2) {
  const unsigned FULL = 0xffffffffu;
  r1 = p1;
  r2 = p2;
  // refine2d_values' test
  const bool inside = (p1 + 1 > 1 + g.tlf1) && (p2 + 1 > 1 + g.tlf2) && (p1 + 1 < 1 + 2 * a.SM1 - g.brb1) &&
                      (p2 + 1 < 1 + 2 * a.SM2 - g.brb2);
  if (!inside) return;
  const double v = lane < 9 ? sim(p1 - 1 + lane % 3, p2 - 1 + lane / 3) : 0.0;
  double mn = __shfl_sync(FULL, v, 0);
#pragma unroll
  for (int k = 0; k < 9; ++k) mn = nmin(mn, __shfl_sync(FULL, v, k));
  // the fit's five values sit on lanes 4 (peak), 3, 5 (along dim 1), 1, 7 (along dim 2)
  const double lg = lane < 9 ? log(1.0 + v - mn) : 0.0;
  const double l[5] = {__shfl_sync(FULL, lg, 4), __shfl_sync(FULL, lg, 3), __shfl_sync(FULL, lg, 5),
                       __shfl_sync(FULL, lg, 1), __shfl_sync(FULL, lg, 7)};
  refine2d_from_logs(p1, p2, l, r1, r2);
}

template <int ALG, int LWN, typename CC>
__device__ __forceinline__ void finish_refine(const Piv2dArgs& a, const IAGeom& g, const IAScalars& sc, int p1, int p2,
                                              int lane, double scale, CC cc, const double* lw, double& r1, double& r2) {
  finish_refine_with(
      a, g, p1, p2, lane,
      [&](int s1, int s2) { return finish_one<ALG, LWN>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale, 0.0, lw); }, r1, r2);
}

#endif  // __CUDACC__

}  // namespace mqp
