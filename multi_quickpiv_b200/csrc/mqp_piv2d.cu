// sm_100a kernels of the 2D path: the fused per-interrogation-area
// correlation / peak kernel (see mqp_piv2d.cuh).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <string>

#include "mqp_finish.cuh"
#include "mqp_internal.h"
#include "mqp_stage.cuh"

namespace mqp {

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
int piv2d_fft_len(int SS1, int SS2) {
  const int SS = SS1 > SS2 ? SS1 : SS2;
  if (SS <= 32) return 32;
  if (SS <= 64) return 64;
  if (SS <= 128) return 128;  // block kernel, mqp_piv2d_big.cu
  return 0;
}

int device_sm_count(int device) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  return n;
}

// Tensor map of an H x W column-major FP32 image for the staged windows of
// FFT length N: dim 0 = rows (contiguous), dim 1 = columns, box (N + 4) x N,
// zero fill outside the image.  False when the image does not qualify (row
// pitch not a multiple of 16 bytes, base not 16-byte aligned) or the driver
// entry point is missing; the caller then launches the unstaged kernel.
bool stage_tensor_map(CUtensorMap* m, const void* img, long long H, long long W, int N) {
  if (H % 4 != 0 || ((uintptr_t)img & 15) != 0 || H < 1 || W < 1) return false;
  typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  // looked up once (thread-safe static initialisation: serving launches from several threads)
  static const EncodeTiled encode = []() -> EncodeTiled {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (EncodeTiled)fn;
    return nullptr;
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)H, (cuuint64_t)W};
  const cuuint64_t strides[1] = {(cuuint64_t)H * 4};
  const cuuint32_t box[2] = {(cuuint32_t)(N + 4), (cuuint32_t)N};
  const cuuint32_t estr[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(img), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Staged windows are on unless MQP_TUNE_PIV2D_TMA=0 (both kernels give
// identical results; the knob exists for timing comparisons).
bool stage_enabled() {
  const char* v = getenv("MQP_TUNE_PIV2D_TMA");  // read per launch: a test may switch it between calls
  return !(v && v[0] == '0');
}

// ZNCC whose interrogation window is half the FFT length in both axes: the
// warp kernel forms the window sums on chip and reads no integral image of
// img2^2 (lw_rows / lw_cols).  Measured on B200 (2048^2 vortex, interSize 32,
// margin 16, step 8, whole pass): ZNCC 2.91 -> 2.77 ms, since it drops eight
// integral-image loads per lag; NSQECC, with four, ran 2.42 -> 2.54 ms (the
// window's second read from L2 costs more than the lookups it replaces), so
// NSQECC keeps the integral image.
bool piv2d_local_sums(int IS1, int IS2, int SM1, int SM2, int alg) {
  if (alg != ALG_ZNCC) return false;
  if (direct2d_ok(IS1, IS2, SM1, SM2)) return false;
  const int N = piv2d_fft_len(IS1 + 2 * SM1, IS2 + 2 * SM2);
  if (N != 32 && N != 64) return false;
  if (piv2d_team_ok(N, true, alg)) return false;
  return IS1 == N / 2 && IS2 == N / 2;
}

int piv2d_warp_f2_lw(int N, int P1, int P2) {
  return N == 64 ? Layout2d<64, true>::warp_f2_lw(P1, P2) : Layout2d<32, true>::warp_f2_lw(P1, P2);
}

int piv2d_warp_f2(int N, bool prune, int P1, int P2, bool masked) {
  if (!masked && piv2d_team_ok(N, prune, ALG_NSQECC)) return piv2d_team_f2(N, P1, P2);
  if (N == 128) return piv2d_big_warp_f2(prune, P1, P2, masked);
  if (N == 64) return prune ? Layout2d<64, true>::warp_f2(P1, P2, masked) : Layout2d<64, false>::warp_f2(P1, P2, masked);
  if (N == 32) return prune ? Layout2d<32, true>::warp_f2(P1, P2, masked) : Layout2d<32, false>::warp_f2(P1, P2, masked);
  return 0;
}

cudaError_t launch_piv2d_batch(const Piv2dBatch& b, cudaStream_t s, std::string& err) {
  if (b.total <= 0 || b.n_items <= 0) return cudaSuccess;
  if (b.N == 128) return launch_piv2d_big_batch(b, s, err);
  if (b.N == 1) return launch_piv2d_direct_batch(b, s, err);
  if (piv2d_team_ok(b.N, b.prune, b.alg)) return launch_piv2d_team_batch(b, s, err);
  if (b.N == 64) return launch_piv2d_b64(b, s, err);
  if (b.N == 32) return launch_piv2d_b32(b, s, err);
  err = "search window larger than 64 along some axis is not supported by the 2D kernel";
  return cudaErrorInvalidValue;
}

bool piv2d_takes_map(const Piv2dArgs& a, int alg) {
  if (alg != ALG_NSQECC && alg != ALG_ZNCC) return false;
  if (direct2d_ok(a.IS1, a.IS2, a.SM1, a.SM2) || piv2d_local_sums(a.IS1, a.IS2, a.SM1, a.SM2, alg)) return false;
  const int N = piv2d_fft_len(a.IS1 + 2 * a.SM1, a.IS2 + 2 * a.SM2);
  if (N && piv2d_team_ok(N, a.IS1 <= N / 2 && a.IS2 <= N / 2, alg)) return false;
  // with SN every lag is formed in full, and only the strip kernel reads a map
  // for that; with planes none does
  if (a.planes || (a.SN && !piv2d_strip_ok(a, alg))) return false;
  // The map costs a pass over all window positions and saves each lag reads of
  // the integral images.  It pays from some number of lags per position.  Whole
  // passes at 2048^2 (an image against itself moved, plus noise) without and with it, us,
  // next to the line:
  //   NSQECC, length 32 (IS 16, SM 8): 0.5 lags 153, 157; 0.7 lags 177, 177; 1.1 lags 239, 223
  //           length 64 (IS 32, SM 16): 0.27 lags 126, 136; 0.48 lags 167, 169; 0.67 lags 207, 201
  //           length 128 (IS 64, SM 32): 0.26 lags 195, 203; 0.44 lags 267, 263; 1.0 lags 400, 378
  //           length 256 (IS 128, SM 64): 1.0 lags 578, 552; 3.8 lags 1682, 1623
  //           with SN (IS 32, SM 16): 1.06 lags 258, 246; 1.4 lags 358, 259
  //   ZNCC,   length 64 (IS 24, SM 16): 0.26 lags 232, 249; 0.48 lags 285, 292; 0.67 lags 340, 334
  //           length 128: 0.26 lags 296, 312; 0.44 lags 379, 379; 1.0 lags 522, 503
  // And on a small image, whatever the number of areas, where one area's walk
  // saves more time than the map takes: a thread's lags beyond the first few
  // hide no latency, some 65,000 positions' worth each.  NSQECC IS 32, SM 16, step 48:
  // 512^2 71, 63; 1024^2 77, 73; 1440^2 91.5, 89.6; SM 10, step 32: 512^2 58.6, 59.3 (58.5, 56.8 in another
  // run); 768^2 67.7, 66.6 (59.0, 60.9); IS 16, SM 8, step 16: 256^2 56.7, 59.4; 640^2 56.7, 59.6; IS 64, SM 32,
  // step 96: 640^2 97, 91; 1024^2 103, 99; 1440^2 125, 146; ZNCC IS 24, SM 16, step 48: 768^2 115, 113; 1440^2 173, 183.
  const double least = a.SN ? 1.0 : (N == 32 ? 0.8 : 0.5);
  const double area_lags = (double)(2 * a.SM1 + 1) * (2 * a.SM2 + 1);
  const double thread_lags = area_lags / (N == 32 || N == 64 ? 32 : (N == 128 ? 128 : 256));
  const double positions = (double)winmap_ld(a.H, a.IS1, a.SM1) * winmap_ld(a.W, a.IS2, a.SM2);
  return positions <= 65536.0 * (thread_lags - 9.0) || area_lags * (double)(a.ia_end - a.ia_begin) >= least * positions;
}

cudaError_t launch_piv2d(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err) {
  if (direct2d_ok(a.IS1, a.IS2, a.SM1, a.SM2)) return launch_piv2d_direct(a, alg, s, err);
  const int SS1 = a.IS1 + 2 * a.SM1, SS2 = a.IS2 + 2 * a.SM2;
  const int N = piv2d_fft_len(SS1, SS2);
  const bool prune = (a.IS1 <= N / 2) && (a.IS2 <= N / 2);
  if (piv2d_team_ok(N, prune, alg)) return launch_piv2d_team(a, N, alg, s, err);
  if (piv2d_strip_ok(a, alg)) return launch_piv2d_strip(a, alg, s, err);
  if (N == 64) return launch_piv2d_w64(a, alg, prune, s, err);
  if (N == 32) return launch_piv2d_w32(a, alg, prune, s, err);
  if (N == 128) return launch_piv2d_big(a, alg, s, err);
  err = "search window larger than 128 along some axis is not supported by the 2D kernels";
  return cudaErrorInvalidValue;
}

}  // namespace mqp
