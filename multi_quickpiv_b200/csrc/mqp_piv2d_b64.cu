// Work-queue (batch) 2D warp kernels at FFT length 64.
#include "mqp_piv2d_warp.cuh"

namespace mqp {

cudaError_t launch_piv2d_b64(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  if (b.lw) return launch_batch_lw<64, 2>(b, s, err);
  return b.prune ? launch_batch_dt<64, true>(b, s, err) : launch_batch_dt<64, false>(b, s, err);
}

}  // namespace mqp
