// Single-pair 2D warp kernels at FFT length 32.
#include "mqp_piv2d_warp.cuh"

namespace mqp {

cudaError_t launch_piv2d_w32(const Piv2dArgs& a, int alg, bool prune, cudaStream_t s, std::string& err) {
  if (piv2d_local_sums(a.IS1, a.IS2, a.SM1, a.SM2, alg)) return launch_lw<32, 3>(a, alg, s, err);
  cudaError_t e = cudaSuccess;
  if (prune ? launch_stg<32, true, 4, 3>(a, alg, s, err, e) : launch_stg<32, false, 4, 3>(a, alg, s, err, e))
    return e;
  // length 32 needs fewer registers: three blocks per SM (12 warps) without spill
  return prune ? launch_dt<32, true, 4, 3>(a, alg, s, err) : launch_dt<32, false, 4, 3>(a, alg, s, err);
}

}  // namespace mqp
