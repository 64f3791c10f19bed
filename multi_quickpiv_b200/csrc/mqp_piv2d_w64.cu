// Single-pair 2D warp kernels at FFT length 64.
#include "mqp_piv2d_warp.cuh"

namespace mqp {

cudaError_t launch_piv2d_w64(const Piv2dArgs& a, int alg, bool prune, cudaStream_t s, std::string& err) {
  if (piv2d_local_sums(a.IS1, a.IS2, a.SM1, a.SM2, alg)) return launch_lw<64, 2>(a, alg, s, err);
  cudaError_t e = cudaSuccess;
  if (prune ? launch_stg<64, true, 4, 2>(a, alg, s, err, e) : launch_stg<64, false, 4, 2>(a, alg, s, err, e))
    return e;
  return prune ? launch_dt<64, true, 4, 2>(a, alg, s, err) : launch_dt<64, false, 4, 2>(a, alg, s, err);
}

}  // namespace mqp
