// Host side of the peak walk (mqp_finish.cuh): the per-lag approximations and
// their open flag, compiled for the CPU.
#include <math.h>

#include "mqp_finish.cuh"

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
