// Host side of the peak walk (mqp_finish.cuh, mqp_finish3.cuh) - the per-lag
// approximations and their open flag, the merges of partial results, the lags
// a window-sum map holds - and of the 256-point kernel's tiles
// (mqp_piv2d_huge.cuh), compiled for the CPU.
#include <math.h>

#include <vector>

#include "mqp_finish3.cuh"
#include "mqp_piv2d_huge.cuh"

#define EMU_API extern "C" __attribute__((visibility("default")))

using namespace mqp;

// Every lag's approximation and similarity_value, and whether any lag is open
// (1) - scale 1, so c is the correlation itself.
EMU_API int mqp_walk_nsqecc(int n, const double* S2, const float* c, double F2, double* walk, double* full) {
  const float sqF = sqrtf((float)F2);
  int open = 0;
  for (int i = 0; i < n; ++i) {
    walk[i] = nsqecc_walk((float)S2[i], sqrtf((float)S2[i]), c[i], -2.f, (float)F2, sqF, open);
    full[i] = similarity_value<ALG_NSQECC>(IAScalars{F2, 0.0, 0.0}, sqF, (double)c[i], S2[i], 0.0, 0.0);
  }
  return open < 0;
}

// The same for masked NSQECC, c1 = (F*mask)*G and S2 = mask*G^2; returns the
// largest magnitude.
EMU_API float mqp_walk_masked(int n, const double* S2, const double* c1, double F2, double* walk, double* full) {
  const float sqF = sqrtf((float)F2);
  float most = 0.f;
  for (int i = 0; i < n; ++i) {
    walk[i] = masked_walk(S2[i], c1[i], F2, sqF, most);
    full[i] = similarity_value<ALG_MASK_NSQECC>(IAScalars{F2, 0.0, 0.0}, sqF, c1[i], S2[i], 0.0, 0.0);
  }
  return most;
}

// Two largest values and the index of the largest over n values split into
// groups of `lanes` (top_take), merged one after the other (top_merge).
EMU_API void mqp_walk_top(int n, int lanes, const float* v, float* b1, float* b2, int* idx) {
  TopTwo all;
  all.b1 = all.b2 = 0.f;
  all.idx = -1;
  for (int l = 0; l < lanes; ++l) {
    TopTwo t;
    t.b1 = t.b2 = 0.f;
    t.idx = -1;
    for (int i = l; i < n; i += lanes) top_take(t, v[i], i);
    top_merge(all, t.b1, t.b2, t.idx);
  }
  *b1 = all.b1;
  *b2 = all.b2;
  *idx = all.idx;
}

// Marks in hit[s1 + P1 s2] the lags of the box that the walk leaves to
// unmapped_at; returns their count.
EMU_API int mqp_walk_unmapped(int lo1, int hi1, int lo2, int hi2, int e1, int e2, int P1, int* hit) {
  LagRanges R{lo1, hi1, lo2, hi2, hi1 - 1, hi2 - 1};
  const UnmappedLags u = unmapped_lags(R, e1, e2);
  for (int q = 0; q < u.count(); ++q) {
    int s1, s2;
    u.at(R, q, s1, s2);
    hit[s1 + P1 * s2] += 1;
  }
  return u.count();
}

// One axis of an IA: its lag box [lo, hi], the last lag whose window sum the
// map holds, and for every lag the window's range and the map's (index in the
// map, first and last image row).
EMU_API void mqp_walk_axis(int v, int st, int IS, int SM, int size, int d, int* box, int* window, int* map) {
  int ir, g0, lo, hi, tlf, brb;
  axis_geom(v, st, IS, SM, size, d, ir, g0, lo, hi, tlf, brb);
  box[0] = tlf;
  box[1] = 2 * SM - brb;
  box[2] = lag_mapped_max(SM, IS, g0, hi, size);
  box[3] = winmap_ld(size, IS, SM);
  for (int s = 0; s <= 2 * SM; ++s) {
    lag_window(s, IS, g0, lo, hi, window[2 * s], window[2 * s + 1]);
    const int i = g0 + s;
    map[3 * s] = i + SM;
    map[3 * s + 1] = i > 0 ? i : 0;
    map[3 * s + 2] = i + IS < size ? i + IS : size;
  }
}

// Stage B of the 256-point kernel over one IA's row spectra: through the tiles,
// thread by thread between the barriers (tiled), or straight from the slot; then
// stage C from the tile or the slot.  G: 128 x 256, F: 128 x 128 float2; lag: P1 P2
// values.
EMU_API void mqp_huge_columns(const float* G, const float* F, int P1, int P2, int tiled, float* lag) {
  const float2* GS = reinterpret_cast<const float2*>(G);
  const float2* FS = reinterpret_cast<const float2*>(F);
  std::vector<float2> sm((size_t)HugeSmem::TOTAL), LG((size_t)P1 * MH), ys((size_t)HUGE_THREADS * QH), fs(ys.size());
  float2 *park = sm.data(), *ft = park + HugeSmem::FT, *pack = park + HugeSmem::PARK, *tw = pack + HugeSmem::PACK;
  for (int j = 0; j < NH; ++j) tw[j] = twiddle_rt(j * (TW_N / NH));
  auto row = [&](std::vector<float2>& v, int t) -> float2(&)[QH] { return *reinterpret_cast<float2(*)[QH]>(&v[(size_t)t * QH]); };
  for (int r = 0; r < 2; ++r) {
    if (tiled) {
      for (int t = 0; t < HUGE_THREADS; ++t) huge_b_tiles(r, t, GS, FS, park, ft);
      for (int t = 0; t < HUGE_THREADS; ++t) huge_b_g(t, park, tw, row(ys, t));
      for (int t = 0; t < HUGE_THREADS; ++t) huge_b_f(r, t, row(ys, t), ft, tw, park, pack, row(fs, t));
    } else {
      for (int t = 0; t < HUGE_THREADS; ++t) huge_b_part1(r, t, GS, FS, tw, park, pack, row(fs, t));
    }
    for (int t = 0; t < HUGE_THREADS; ++t) huge_b_part2(r, t, tw, park, pack, row(fs, t));
    for (int t = 0; t < HUGE_THREADS; ++t) huge_b_part3(r, t, P1, park, LG.data());
  }
  if (tiled && huge_c_tiled(P1)) {
    for (int t = 0; t < HUGE_THREADS; ++t) huge_c_tile(t, P1, LG.data(), park);
    for (int s1 = 0; s1 < P1; ++s1)
      for (int h = 0; h < 2; ++h) huge_lag_row(s1, h, P1, P2, park, lag, 1.f, HugeSmem::LS);
  } else {
    for (int s1 = 0; s1 < P1; ++s1)
      for (int h = 0; h < 2; ++h) huge_lag_row(s1, h, P1, P2, LG.data(), lag, 1.f);
  }
}

// packed_product over the 2M bins of two real rows' spectra in one column
EMU_API void mqp_packed_column(int M, const float* G, const float* F, float* out) {
  const float2 *g = reinterpret_cast<const float2*>(G), *f = reinterpret_cast<const float2*>(F);
  for (int h = 0; h < 2; ++h)
    for (int m = 0; m < M; ++m) {
      const int k = 2 * m + h, kn = 2 * packed_mirror(M, h, m) + h;
      reinterpret_cast<float2*>(out)[k] = packed_product(g[k], g[kn], f[k], f[kn]);
    }
}
