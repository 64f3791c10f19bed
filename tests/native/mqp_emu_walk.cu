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
