// The 3D finish without the full similarity of every lag (mqp_finish.cuh gives
// the 2D one and the error bounds the gap rests on: the similarity's formula
// is the same), and its window-sum maps: ws / wz[(i + SM1) + ldw1 ((j + SM2) + ldw2
// (k + SM3))] hold the sums over the interrogation-sized window at (i, j, k)
// clipped to the volume, in box_sum3's order.
#pragma once

#include "mqp_finish.cuh"
#include "mqp_piv3d.cuh"

namespace mqp {

// One block's share of an IA's lags: its two largest values and the lag of the
// largest (FFTCC: exact, the lowest index of equal ones).
struct TopPart3 {
  float b1, b2;
  int idx, pad_;
};
static_assert(sizeof(TopPart3) <= sizeof(PeakPart3), "shares the parts' scratch");

// The pass ends in the walk: no SN, no planes, one of the unmasked similarities.
MQP_HD MQP_FI bool finish3_fast(const Piv3dArgs& a, int alg) {
  return a.SN == nullptr && a.planes == nullptr && alg != ALG_MASK_NSQECC;
}

// two partial results into one
MQP_HD MQP_FI void top_merge(TopTwo& t, float o1, float o2, int oi) {
  if (o1 > t.b1 || (o1 == t.b1 && oi >= 0 && (t.idx < 0 || oi < t.idx))) {
    t.b2 = t.b1 > o2 ? t.b1 : o2;
    t.b1 = o1;
    t.idx = oi;
  } else if (o1 > t.b2) {
    t.b2 = o1;
  }
}

// Similarity of lag (s1, s2, s3) in full from its raw correlation c, as
// k3c_pair forms it.
template <int ALG>
MQP_HD MQP_FI double full_sim3(const Piv3dArgs& a, const IAGeom3& g, const IA3State& s, int s1, int s2, int s3,
                               double c) {
  if (ALG == ALG_FFTCC) return c;
  const float sqF = sqrtf((float)s.sumF2);
  int r0, r1, c0, c1, z0, z1;
  lag_window(s1, a.IS[0], g.g0[0], g.lo[0], g.hi[0], r0, r1);
  lag_window(s2, a.IS[1], g.g0[1], g.lo[1], g.hi[1], c0, c1);
  lag_window(s3, a.IS[2], g.g0[2], g.lo[2], g.hi[2], z0, z1);
  const double S2 = box_sum3(a.IIg2, a.H, a.W, r0, r1, c0, c1, z0, z1);
  double S1 = 0.0, n = 0.0;
  if (ALG == ALG_ZNCC) {
    S1 = box_sum3(a.IIg, a.H, a.W, r0, r1, c0, c1, z0, z1);
    n = (double)(r1 - r0) * (double)(c1 - c0) * (double)(z1 - z0);
  }
  return similarity_value<ALG>(IAScalars{s.sumF2, s.meanF, s.meanG}, sqF, c, S2, S1, n);
}

}  // namespace mqp
