// Work-queue (batch) 2D warp kernels at FFT length 32.
#include "mqp_piv2d_warp.cuh"

namespace mqp {

cudaError_t launch_piv2d_b32(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  if (b.lw) return launch_batch_lw<32, 3>(b, s, err);
  return b.prune ? launch_batch_dt<32, true>(b, s, err) : launch_batch_dt<32, false>(b, s, err);
}

}  // namespace mqp
