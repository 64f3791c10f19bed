// Strip kernel: FFTCC and NSQECC passes whose neighbouring interrogation areas
// (IAs) overlap, at FFT length 64 with interrogation windows up to 32.
//
// IAs above one another (consecutive along dim 1, same columns) read the same
// pixel rows through the same columns, so a row's transform along dim 2 is
// the same for all of them.  A block takes a strip of n IAs: its warps
// transform every image row the strip's windows touch once, into shared
// memory, and then each IA's warp works through that IA alone - columns
// (forward G, forward F, product, inverse), lag rows, peak, fit - reading
// the shared row spectra at the IA's own offset.  At step 8 a strip of four
// transforms 36 rows per IA instead of 96.
//
// The spectra being shared and read-only, a warp cannot park its column's G
// spectrum and its first half inverse in its own copy of the rows, as the
// one-warp-per-IA kernel (mqp_piv2d_warp.cuh) does: they wait in tensor
// memory (tcgen05.st / tcgen05.ld, 128 columns per block), which leaves the
// registers to one transform at a time.  The lag spectra and the correlation
// plane take the rows' place in shared memory once the block is through with
// them, so a block needs 42 KB at step 8 and three blocks, twelve warps, fit on
// an SM, where the other kernel's 26 KB per warp and 255 registers fit eight
// warps.  (A block takes up to 81 KB; past 75 KB - interSize 32, margin 16, from
// step 29 - two blocks fit.)  Each correlation and similarity goes through the
// same operations in the same order as there, so the vectors are the same bit
// for bit; SN's FP64 sum over the lags runs in another order.
//
// Bound by instruction issue and supply (ncu, 1024^2 NSQECC step 8): 11.7k warp
// instructions per IA (15.3k before), issue active 54 %, stalls led by
// wait (0.93 warps per issue) and no_instruction (0.91).  Measured on B200 (kernel,
// one warp per IA -> strips): 2048^2 NSQECC step 8 2113 -> 1202 us, FFTCC 1270 ->
// 1023; 1024x1280 NSQECC step 16 199 -> 93; 2048^2 NSQECC step 16 with SN 589 ->
// 354; 256^2 FFTCC Float64 step 16 35 -> 17.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "mqp_finish.cuh"
#include "mqp_internal.h"

namespace mqp {

namespace {

constexpr int SN_ = 64;            // FFT length
constexpr int SM_ = SN_ / 2;       // spectrum columns per IA: one per lane
// Four warps, three blocks to an SM (168 registers): twelve warps.  Measured on
// the 2048^2 NSQECC pass at step 8: 1403 us so, 1775 with four (128 registers,
// 1.5 KB of spill), 1592 with two (255 registers, no spill), 1653 with one
// block of eight warps and IAs (all before the rows loaded in batches); block
// sizes that are not a multiple of four warps load the SM's quarters unevenly.
constexpr int STRIP_WARPS = 4, STRIP_BLOCKS = 3;

// Shared-memory layout of a block (float2 units unless said otherwise) and
// the strip's shape.
struct StripCfg {
  int n;        // IAs of a strip
  int wpi;      // warps per IA through the columns (1, or 2: one per half spectrum)
  int strips;   // strips per IA column
  int v2_0;     // first IA column
  int rsg, rsf; // row-spectrum strides of G and F (odd: lanes over columns hit distinct banks)
  int ps;       // stride of a warp's private rows
  int off_f, off_priv, off_tail, off_red, off_tw, off_pk;
  int priv;     // float2 per IA
  int tail;     // float2 per IA
  size_t bytes;
};

MQP_HD MQP_FI float2 dif_odd(float2 a, float2 b, float2 w) {  // (a - b) conj(w), as split_G_pair
  const float2 d = csub(a, b);
  return make_float2(d.x * w.x + d.y * w.y, d.y * w.x - d.x * w.y);
}

__device__ __forceinline__ double sum32(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double max32(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ void pair_barrier(int id) {
#if defined(__CUDA_ARCH__)
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
#else
  (void)id;
#endif
}

// Row `row` of the strip's G rows (image row Rg0 + row, the search window's
// columns, zero outside them) or F rows (image row ir1 + row): its r2c along
// dim 2.  F rows leave the maximum and the FP64 sum of squares of their
// pixels.  The sums of row_process, value by value.
template <typename T>
__device__ __forceinline__ void strip_row(const Piv2dArgs& a, const IAGeom& g, bool isF, long long base, float2* out,
                                          int stride, double2* red) {
  // loads in batches at addresses clamped into the row, before any is used: one
  // by one under their conditions they cost a round trip each (2048^2 NSQECC
  // step 8 1403 -> 1202 us, step 16 with SN 432 -> 354)
  float2 z[SM_];
  const long long H = a.H;
  constexpr int RB = SM_;
  if (isF) {
    const T* p = reinterpret_cast<const T*>(a.img1) + base;
    const int IS2 = a.IS2;
    T raw[RB];
#pragma unroll
    for (int x = 0; x < RB; ++x) raw[x] = ldg_px<T>(p, H * (x < IS2 ? x : IS2 - 1));
    mqp_no_hoist();
    double vmax = -INFINITY, sumsq = 0.0;
#pragma unroll
    for (int x = 0; x < RB; ++x) {
      float w = 0.f;
      if (x < IS2) {
        const double val = (double)raw[x];
        vmax = val > vmax ? val : vmax;
        sumsq += val * val;
        w = (float)val;
      }
      if (x & 1) z[x / 2].y = w;
      else z[x / 2].x = w;
    }
#pragma unroll
    for (int n = RB / 2; n < SM_; ++n) z[n] = make_float2(0.f, 0.f);
    *red = make_double2(vmax, sumsq);
  } else {
    const T* p = reinterpret_cast<const T*>(a.img2) + base;
    const int lo2 = g.lo2, hi2 = g.hi2;
#pragma unroll
    for (int b = 0; b < SN_; b += RB) {
      T raw[RB];
#pragma unroll
      for (int x = 0; x < RB; ++x) {
        const int c = b + x < lo2 ? lo2 : (b + x < hi2 ? b + x : hi2 - 1);
        raw[x] = ldg_px<T>(p, H * c);
      }
      if (sizeof(T) == 8) mqp_no_hoist();
#pragma unroll
      for (int x = 0; x < RB; ++x) {
        const float v = (b + x >= lo2 && b + x < hi2) ? (float)raw[x] : 0.f;
        if (x & 1) z[(b + x) / 2].y = v;
        else z[(b + x) / 2].x = v;
      }
    }
  }
  r2c_store<SN_, SM_>(z, out, stride);
}

// Tensor memory as a warp's register park: 64 columns hold one half spectrum
// (32 float2 per lane) while another transform has the registers.  Each warp
// of the block uses its own 32 lanes of the block's columns.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {  // one warp
#if defined(__CUDA_ARCH__)
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(slot))
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
#else
  (void)slot;
#endif
}
__device__ __forceinline__ void tmem_free(uint32_t base) {  // the same warp, after every use
#if defined(__CUDA_ARCH__)
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(base));
#else
  (void)base;
#endif
}
// 16 float2 per lane to / from columns [addr, addr + 32)
__device__ __forceinline__ void tmem_put(uint32_t addr, const float2 (&v)[16]) {
#if defined(__CUDA_ARCH__)
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
      "f"(v[0].x), "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y),
      "f"(v[4].x), "f"(v[4].y), "f"(v[5].x), "f"(v[5].y), "f"(v[6].x), "f"(v[6].y), "f"(v[7].x), "f"(v[7].y),
      "f"(v[8].x), "f"(v[8].y), "f"(v[9].x), "f"(v[9].y), "f"(v[10].x), "f"(v[10].y), "f"(v[11].x), "f"(v[11].y),
      "f"(v[12].x), "f"(v[12].y), "f"(v[13].x), "f"(v[13].y), "f"(v[14].x), "f"(v[14].y), "f"(v[15].x), "f"(v[15].y)
      : "memory");
#else
  (void)addr, (void)v;
#endif
}
__device__ __forceinline__ void tmem_put_wait() {
#if defined(__CUDA_ARCH__)
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#endif
}
// The wait names the registers it guards, so that no use moves above it.
__device__ __forceinline__ void tmem_get(uint32_t addr, float2 (&v)[16]) {
#if defined(__CUDA_ARCH__)
  asm volatile(
      "{\n tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      " tcgen05.wait::ld.sync.aligned;\n}"
      : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x), "=f"(v[3].y),
        "=f"(v[4].x), "=f"(v[4].y), "=f"(v[5].x), "=f"(v[5].y), "=f"(v[6].x), "=f"(v[6].y), "=f"(v[7].x), "=f"(v[7].y),
        "=f"(v[8].x), "=f"(v[8].y), "=f"(v[9].x), "=f"(v[9].y), "=f"(v[10].x), "=f"(v[10].y), "=f"(v[11].x), "=f"(v[11].y),
        "=f"(v[12].x), "=f"(v[12].y), "=f"(v[13].x), "=f"(v[13].y), "=f"(v[14].x), "=f"(v[14].y), "=f"(v[15].x), "=f"(v[15].y)
      : "r"(addr)
      : "memory");
#else
  (void)addr;
  for (int i = 0; i < 16; ++i) v[i] = make_float2(0.f, 0.f);
#endif
}

// conj of conj(F^) G^ over one half spectrum (stage_product): t = F^ in fpos
// slots on entry, G^ in the warp's tensor memory in the same order.  Lane 0
// holds the packed pair of real columns (k2 = 0 and 32), whose bins k and -k
// have to be taken apart: it leaves its bins in pk (96 float2) and every lane
// forms one of the products; alone, lane 0 would take the other lanes through
// some 500 instructions.
__device__ __forceinline__ void strip_product(int lane, int h, uint32_t tm, float2 (&t)[SM_], float2* pk) {
  constexpr int M = SM_;
  float2 p[M];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float2 x[16];
    tmem_get(tm + 32 * q, x);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int j = fpos<M>(m);
      if (j / 16 != q) continue;
      const float2 f = t[j], g = x[j - 16 * q];
      if (lane == 0) {
        pk[m] = g;
        pk[M + m] = f;
      }
      p[m] = cconj(cmulc(f, g));
    }
  }
  __syncwarp();
  {
    const int mm = packed_mirror(M, h, lane);
    pk[2 * M + lane] = cconj(packed_product(pk[lane], pk[mm], pk[M + lane], pk[M + mm]));
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < M; ++m) t[m] = p[m];
  if (lane == 0) {
#pragma unroll
    for (int m = 0; m < M; ++m) t[m] = pk[2 * M + m];
  }
}

// Peak (first_fullovp_peak), SN and Gaussian fit of one IA from its plane (rows
// below 32) and tail rows.  Not inlined: the transforms before it have the
// registers to themselves.
template <int ALG, bool SN>
__device__ __noinline__ void strip_finish(const Piv2dArgs& a, int v1, int v2, double sumF2, const float* plane,
                                          const float* tailp, int lane) {
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1, lane_rows = P1 < 32 ? P1 : 32;
  const IAGeom g = ia_geom(a, v1, v2);
  const long long vfo = (long long)v1 + (long long)a.vf1 * v2;
  IAScalars sc;
  sc.meanF = sc.meanG = 0.0;
  sc.sumF2 = sumF2;
  const double scale = cc_scale<SN_>();
  auto cc = [&](int s1, int s2) {
    return s1 < lane_rows ? plane[s1 * P2 + s2] : tailp[(s1 - lane_rows) * P2 + s2];
  };
  LagRanges R;
  R.lo1 = g.tlf1;
  R.hi1 = 2 * a.SM1 - g.brb1;
  R.lo2 = g.tlf2;
  R.hi2 = 2 * a.SM2 - g.brb2;
  R.shi1 = 2 * a.SM1 - 1 - g.brb1;
  R.shi2 = 2 * a.SM2 - 1 - g.brb2;
  int bidx = -1;
  double sn = 0.0;
  if (SN) {
    // the similarities are FP32 values (FFTCC: before the transforms' scale),
    // so peak and maximum compare in FP32; only the sum is FP64
    float best = 0.f, smax = -INFINITY;
    double ssum = 0.0;
    auto take = [&](int s1, int s2, float v) {
      if (v > best || (v == best && s1 + P1 * s2 < bidx)) {
        best = v;
        bidx = s1 + P1 * s2;
      }
      if (s1 <= R.shi1 && s2 <= R.shi2) {
        smax = (v > smax || v != v) ? v : smax;
        ssum += ALG == ALG_FFTCC ? (double)v * scale : (double)v;
      }
    };
    if (ALG == ALG_FFTCC) {
      if (lane < lane_rows && lane >= R.lo1 && lane <= R.hi1)
        for (int s2 = R.lo2; s2 <= R.hi2; ++s2) take(lane, s2, cc(lane, s2));
      for (int s1 = lane_rows > R.lo1 ? lane_rows : R.lo1; s1 <= R.hi1; ++s1)
        for (int s2 = R.lo2 + lane; s2 <= R.hi2; s2 += 32) take(s1, s2, cc(s1, s2));
    } else if (a.wd) {
      const int e1 = min(lag_mapped_max(a.SM1, a.IS1, g.g01, g.hi1, a.H), R.hi1);
      const int e2 = min(lag_mapped_max(a.SM2, a.IS2, g.g02, g.hi2, a.W), R.hi2);
      // similarity_value with the square root and the FP64 sum of the map
      const float sqF = sqrtf((float)sc.sumF2);
      const long long w0 = (g.g01 + a.SM1) + (long long)a.ldw * (g.g02 + a.SM2);
      auto sim = [&](float q, double S2, float c) {
        const float d = q * sqF;
        const double n = (sc.sumF2 - 2.0 * ((double)c * scale)) + S2;
        return d / (float)(n + (double)d);
      };
      constexpr int B = 8;  // lags whose sums are loaded before any is used
      if (lane < lane_rows && lane >= R.lo1 && lane <= e1) {
        for (int b = R.lo2; b <= e2; b += B) {
          double S2[B];
          float q[B];
#pragma unroll
          for (int k = 0; k < B; ++k) {  // past the box: the last column again, not taken
            const long long w = w0 + lane + (long long)a.ldw * min(b + k, e2);
            S2[k] = __ldg(a.wd + w);
            q[k] = __ldg(&a.ws[w].y);
          }
          mqp_no_hoist();
#pragma unroll
          for (int k = 0; k < B; ++k)
            if (b + k <= e2) take(lane, b + k, sim(q[k], S2[k], cc(lane, b + k)));
        }
      }
      for (int s1 = lane_rows > R.lo1 ? lane_rows : R.lo1; s1 <= e1; ++s1)
        for (int s2 = R.lo2 + lane; s2 <= e2; s2 += 32) {
          const long long w = w0 + s1 + (long long)a.ldw * s2;
          take(s1, s2, sim(__ldg(&a.ws[w].y), __ldg(a.wd + w), cc(s1, s2)));
        }
      const UnmappedLags u = unmapped_lags(R, e1, e2);
#pragma unroll 1
      for (int q = lane; q < u.count(); q += 32) {
        int s1, s2;
        u.at(R, q, s1, s2);
        take(s1, s2, (float)finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale));
      }
    } else {
      const int w2 = R.hi2 - R.lo2 + 1, total = (R.hi1 - R.lo1 + 1) * w2;
#pragma unroll 1
      for (int q = lane; q < total; q += 32) {
        const int s1 = R.lo1 + q / w2, s2 = R.lo2 + q % w2;
        take(s1, s2, (float)finish_one<ALG>(a, g, sc, s1, s2, (double)cc(s1, s2) * scale));
      }
    }
    // merged as peak_merge: the largest value, of equal ones the lowest index
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, off), om = __shfl_xor_sync(0xffffffffu, smax, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, off);
      if (oi >= 0 && (bidx < 0 || ob > best || (ob == best && oi < bidx))) {
        best = ob;
        bidx = oi;
      }
      smax = (om > smax || om != om) ? om : smax;
    }
    ssum = sum32(ssum);
    // compute_SN (src/utils/piv_ops.jl:336-367) over [TLF_off, 2SM-1-BRB_off]
    const double top = ALG == ALG_FFTCC ? (double)smax * scale : (double)smax;
    const double len = (double)(R.shi1 - R.lo1 + 1) * (double)(R.shi2 - R.lo2 + 1);
    sn = top / ((ssum - top) / (len - 1.0));
  } else {
    bidx = finish_search<ALG, 32, 0>(a, g, sc, R, lane, P1, scale, cc, nullptr, nullptr);
  }
  double r1 = -1.0, r2 = -1.0;  // no peak: 1-based (0, 0), displacement -(SM+1)
  if (bidx >= 0) finish_refine<ALG, 0>(a, g, sc, bidx % P1, bidx / P1, lane, scale, cc, nullptr, r1, r2);
  if (lane == 0) {
    a.VF[2 * vfo + 0] = r1 - a.SM1;
    a.VF[2 * vfo + 1] = r2 - a.SM2;
    if (SN) a.SN[vfo] = sn;
  }
}

// One IA of the strip, from its rows' spectra to its vector; gA is the strip's
// first IA, Rg0 the image row of the strip's first G row, tm the warp's tensor
// memory.  role: which half spectrum, where two warps share an IA.
template <int ALG, typename T, bool SN>
__device__ __forceinline__ void strip_ia(const Piv2dArgs& a, const StripCfg& c, float2* smem, const IAGeom& gA, int Rg0,
                                         int v1, int v2, int k, int role, int warp, int lane, uint32_t tm) {
  constexpr int N = SN_, M = SM_;
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1;
  const float2* Gs = smem;
  const float2* Fs = smem + c.off_f;
  const double2* red = reinterpret_cast<const double2*>(smem + c.off_red);
  const float2* tw = smem + c.off_tw;
  const IAGeom g = ia_geom(a, v1, v2);
  const long long vfo = (long long)v1 + (long long)a.vf1 * v2;
  IAScalars sc;
  sc.meanF = 0.0;
  sc.meanG = 0.0;
  {
    const double2 rr = lane < a.IS1 ? red[g.ir1 - gA.ir1 + lane] : make_double2(-INFINITY, 0.0);
    const double vmax = max32(rr.x);
    sc.sumF2 = sum32(rr.y);
    // skip_inter_region (src/utils/piv_ops.jl:134-157): the vector stays zero
    if (a.threshold >= 0.0 && vmax < a.threshold) {
      if (role == 0 && lane == 0) {
        a.VF[2 * vfo + 0] = 0.0;
        a.VF[2 * vfo + 1] = 0.0;
        if (SN) a.SN[vfo] = 0.0;
      }
      if (c.wpi == 1) __syncthreads();
      return;
    }
  }
  float2* priv = smem + c.off_priv + k * c.priv;
  float* tailp = reinterpret_cast<float*>(smem + c.off_tail + k * c.tail);
  float2* pk = smem + c.off_pk + warp * 3 * M;
  // lag rows beyond the lanes (P1 = 33..36): a direct sum by the whole warp
  const int lane_rows = P1 < 32 ? P1 : 32;
  {
    const float2* Grow = Gs + lane * c.rsg + (g.g01 - Rg0);
    const float2* Frow = Fs + lane * c.rsf + (g.ir1 - gA.ir1);
    float2* prow = priv + lane * c.ps;
    // window rows that hold data: the others are zero for this IA whatever the strip has there
    const unsigned long long lm = (g.hi1 >= 64 ? ~0ull : (1ull << g.hi1) - 1) & ~((1ull << g.lo1) - 1);
    const unsigned lm0 = (unsigned)lm, lm1 = (unsigned)(lm >> 32);
    const unsigned fm = a.IS1 >= 32 ? ~0u : (1u << a.IS1) - 1;
    const float2 zero = make_float2(0.f, 0.f);
    // the columns (per half spectrum h: the G column, the F column, the
    // inverse of their product), then the lag row, as stages around one copy of
    // the transform: with a copy per stage the warps waited for instructions
    float2 t[M];
    const int j0 = role == 1 ? 3 : 0, j1 = (c.wpi == 2 && role == 0) ? 3 : 7;
#pragma unroll 1
    for (int job = j0; job < j1; ++job) {
      const int h = job >= 3, st = job - 3 * h;
      if (st == 0) {
        // even bins from g[n] + g[n + M], odd from their difference turned; a
        // row without data is not read: it may lie outside the strip
        if (lm == ~0ull) {
          if (h == 0) {
#pragma unroll
            for (int n = 0; n < M; ++n) {
              t[n] = cadd(Grow[n], Grow[n + M]);
              if (n % 8 == 7) mqp_no_hoist();
            }
          } else {
#pragma unroll
            for (int n = 0; n < M; ++n) {
              t[n] = dif_odd(Grow[n], Grow[n + M], tw[n]);
              if (n % 8 == 7) mqp_no_hoist();
            }
          }
        } else {
#pragma unroll
          for (int n = 0; n < M; ++n) {
            const float2 u = (lm0 >> n) & 1u ? Grow[n] : zero, v = (lm1 >> n) & 1u ? Grow[n + M] : zero;
            t[n] = h == 0 ? cadd(u, v) : dif_odd(u, v, tw[n]);
            if (n % 8 == 7) mqp_no_hoist();
          }
        }
      } else if (st == 1) {
#pragma unroll
        for (int n = 0; n < M; ++n) {
          t[n] = (fm >> n) & 1u ? Frow[n] : zero;
          if (n % 8 == 7) mqp_no_hoist();
        }
        if (h) {
#pragma unroll
          for (int n = 1; n < M; ++n) t[n] = rotate<N, false>(t[n], n);
        }
      } else if (st == 3) {
        __syncwarp();
        // the tail rows first, since the plane takes the lag spectra's place
#pragma unroll 1
        for (int s1 = lane_rows; s1 < P1; ++s1) {
          const float2 X0 = priv[s1];
          const int sb = lane + 32;  // each lane's lags: lane, lane + 32 (P2 <= 64)
          float acc = 0.f, accb = 0.f;
          int ti = 0, tb = 0;
#pragma unroll 4
          for (int kk = 1; kk < M; ++kk) {
            ti = (ti + lane) & (N - 1);
            tb = (tb + sb) & (N - 1);
            const float2 X = priv[kk * c.ps + s1];
            const float2 w = tw[ti], wb = tw[tb];
            acc += X.x * w.x - X.y * w.y;
            accb += X.x * wb.x - X.y * wb.y;
          }
          float* trow = tailp + (s1 - lane_rows) * P2;
          if (lane < P2) trow[lane] = X0.x + ((lane & 1) ? -X0.y : X0.y) + 2.f * acc;
          if (sb < P2) trow[sb] = X0.x + ((sb & 1) ? -X0.y : X0.y) + 2.f * accb;
        }
        // lag row s1 = lane: c2r split, conjugated (c2r_pre)
        const float2* col = priv + (lane < lane_rows ? lane : 0);
        const float X0 = col[0].x, XM = col[0].y;
        t[0] = cconj(cadd(make_float2(X0 + XM, 0.f), cmul_pi(make_float2(X0 - XM, 0.f))));
#pragma unroll
        for (int kk = 1; kk <= M / 2; ++kk) {
          const float2 A0 = col[kk * c.ps], A1 = col[(M - kk) * c.ps];
          const float2 B0 = cconj(A1), B1 = cconj(A0);
          t[kk] = cconj(cadd(cadd(A0, B0), cmul_pi(rotate<N, true>(csub(A0, B0), kk))));
          if (kk != M / 2) t[M - kk] = cconj(cadd(cadd(A1, B1), cmul_pi(rotate<N, true>(csub(A1, B1), M - kk))));
          if (kk % 4 == 3) mqp_no_hoist();
        }
        __syncwarp();
      }
      fft_reg<M, false>(t);
      if (st == 0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float2 x[16];
#pragma unroll
          for (int n = 0; n < 16; ++n) x[n] = t[16 * q + n];
          tmem_put(tm + 32 * q, x);
        }
        tmem_put_wait();
      } else if (st == 1) {
        strip_product(lane, h, tm, t, pk);
      } else if (st == 2) {
        // R[s] = A0[s] + W^-s A1[s] and R[s + M] = A0[s] - W^-s A1[s], the
        // lags s < P1 kept.  A0 waits in tensor memory, or in shared memory
        // for the pair's other warp; one warp per IA puts its lag spectra
        // where the rows were, once every warp of the block is through them.
        if (h == 0) {
          if (c.wpi == 2) {
#pragma unroll
            for (int n = 0; n < M; ++n) prow[n] = cconj(t[fpos<M>(n)]);
            pair_barrier(1 + k);
          } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              float2 x[16];
#pragma unroll
              for (int n = 0; n < 16; ++n) x[n] = t[16 * q + n];
              tmem_put(tm + 64 + 32 * q, x);
            }
            tmem_put_wait();
          }
        } else if (c.wpi == 2) {
          pair_barrier(1 + k);
#pragma unroll
          for (int n = 0; n < M; ++n) {
            const float2 a0 = prow[n];
            const float2 r = rotate<N, true>(cconj(t[fpos<M>(n)]), n);
            if (n < P1) prow[n] = cadd(a0, r);
            if (n + M < P1) prow[n + M] = csub(a0, r);
          }
        } else {
          __syncthreads();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float2 x[16];
            tmem_get(tm + 64 + 32 * q, x);
#pragma unroll
            for (int n = 0; n < M; ++n) {
              const int j = fpos<M>(n);
              if (j / 16 != q) continue;
              const float2 a0 = cconj(x[j - 16 * q]);
              const float2 r = rotate<N, true>(cconj(t[j]), n);
              if (n < P1) prow[n] = cadd(a0, r);
              if (n + M < P1) prow[n + M] = csub(a0, r);
            }
          }
        }
      } else if (lane < lane_rows) {
        float* crow = reinterpret_cast<float*>(priv) + lane * P2;
#pragma unroll
        for (int n = 0; n < M; ++n) {
          const float2 z = cconj(t[fpos<M>(n)]);
          if (2 * n < P2) crow[2 * n] = z.x;
          if (2 * n + 1 < P2) crow[2 * n + 1] = z.y;
        }
      }
    }
    if (c.wpi == 2 && role == 0) return;
  }
  __syncwarp();
  strip_finish<ALG, SN>(a, v1, v2, sc.sumF2, reinterpret_cast<const float*>(priv), tailp, lane);
}

template <int ALG, typename T, bool SN>
__global__ void __launch_bounds__(STRIP_WARPS * 32, STRIP_BLOCKS) strip_kernel(const __grid_constant__ Piv2dArgs a, StripCfg c) {
  extern __shared__ __align__(16) float2 smem[];
  constexpr int N = SN_;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int v2 = c.v2_0 + (int)(blockIdx.x / c.strips);
  const int v1a = (int)(blockIdx.x % c.strips) * c.n;
  const int cnt = min(c.n, a.vf1 - v1a);
  float2* Gs = smem;
  float2* Fs = smem + c.off_f;
  double2* red = reinterpret_cast<double2*>(smem + c.off_red);
  float2* tw = smem + c.off_tw;
  __shared__ uint32_t tm_base;
  if (warp == 0) tmem_alloc(&tm_base);
  for (int j = threadIdx.x; j < N; j += blockDim.x) tw[j] = twiddle_rt(j * (TW_N / N));
  const IAGeom gA = ia_geom(a, v1a, v2), gB = ia_geom(a, v1a + cnt - 1, v2);
  const int Rg0 = gA.g01 + gA.lo1, nG = gB.g01 + gB.hi1 - Rg0;
  const int nF = (cnt - 1) * a.st1 + a.IS1;

  // ---- the strip's rows, one per thread: G first, then F ----
#pragma unroll 1
  for (int r = threadIdx.x; r < nG + nF; r += STRIP_WARPS * 32) {
    const bool isF = r >= nG;
    const int row = isF ? r - nG : r;
    const long long base = isF ? (long long)(gA.ir1 + row) + (long long)a.H * gA.ir2
                               : (long long)(Rg0 + row) + (long long)a.H * gA.g02;
    strip_row<T>(a, gA, isF, base, (isF ? Fs : Gs) + row, isF ? c.rsf : c.rsg, red + row);
  }
  __syncthreads();

  // ---- one IA per warp (or pair of warps) ----
  const int k = warp / c.wpi, role = warp - k * c.wpi;
  const uint32_t tm = tm_base + ((uint32_t)(warp & 3) << 21);  // the warp's 32 lanes
  if (k < cnt) strip_ia<ALG, T, SN>(a, c, smem, gA, Rg0, v1a + k, v2, k, role, warp, lane, tm);
  else if (c.wpi == 1) __syncthreads();  // the barrier inside strip_ia
  __syncthreads();
  if (warp == 0) tmem_free(tm_base);
}

StripCfg strip_cfg(const Piv2dArgs& a, int n, int wpi) {
  StripCfg c{};
  const int P1 = 2 * a.SM1 + 1, P2 = 2 * a.SM2 + 1;
  c.n = n;
  c.wpi = wpi;
  c.strips = (a.vf1 + n - 1) / n;
  c.rsg = (a.IS1 + 2 * a.SM1 + (n - 1) * a.st1) | 1;
  c.rsf = (a.IS1 + (n - 1) * a.st1) | 1;
  c.ps = std::max(SM_, P1) | 1;
  c.priv = SM_ * c.ps;
  c.tail = P1 > 32 ? ((P1 - 32) * P2 + 1) / 2 : 0;
  c.off_f = SM_ * c.rsg;
  const int rows = c.off_f + SM_ * c.rsf;
  c.off_priv = wpi == 1 ? 0 : rows;  // over the rows, or beside them
  c.off_tail = wpi == 1 ? std::max(rows, n * c.priv) : rows + n * c.priv;
  c.off_red = (c.off_tail + n * c.tail + 1) & ~1;  // double2: 16-byte aligned
  c.off_tw = c.off_red + 2 * (a.IS1 + (n - 1) * a.st1);
  c.off_pk = c.off_tw + SN_;
  c.bytes = (size_t)(c.off_pk + STRIP_WARPS * 3 * SM_) * sizeof(float2);
  return c;
}

template <int ALG, typename T, bool SN>
cudaError_t strip_launch(const Piv2dArgs& a, const StripCfg& c, cudaStream_t s, std::string& err) {
  auto kern = strip_kernel<ALG, T, SN>;
  cudaError_t e = allow_dyn_smem(kern, c.bytes);
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return e;
  }
  const long long cols = (a.ia_end - a.ia_begin) / a.vf1;
  kern<<<(unsigned)(cols * c.strips), STRIP_WARPS * 32, c.bytes, s>>>(a, c);
  e = cudaGetLastError();
  if (e != cudaSuccess) err = std::string("piv2d strip launch: ") + cudaGetErrorString(e);
  return e;
}

template <int ALG, typename T>
cudaError_t strip_sn(const Piv2dArgs& a, const StripCfg& c, cudaStream_t s, std::string& err) {
  return a.SN ? strip_launch<ALG, T, true>(a, c, s, err) : strip_launch<ALG, T, false>(a, c, s, err);
}

template <int ALG>
cudaError_t strip_dt(const Piv2dArgs& a, const StripCfg& c, cudaStream_t s, std::string& err) {
  return a.dtype == 0 ? strip_sn<ALG, float>(a, c, s, err) : strip_sn<ALG, double>(a, c, s, err);
}

}  // namespace

bool piv2d_strip_ok(const Piv2dArgs& a, int alg) {
  if (alg != ALG_FFTCC && alg != ALG_NSQECC) return false;
  if (a.pred || a.planes) return false;
  if (a.IS1 > SM_ || a.IS2 > SM_ || a.vf1 < 1 || a.st1 > a.IS1) return false;
  if (piv2d_fft_len(a.IS1 + 2 * a.SM1, a.IS2 + 2 * a.SM2) != SN_) return false;
  if (2 * a.SM1 + 1 > 36) return false;  // one lag row per lane, up to four by direct sums
  if (a.ia_begin % a.vf1 != 0 || a.ia_end % a.vf1 != 0) return false;  // whole IA columns
  return (a.ia_end - a.ia_begin) / a.vf1 * (long long)a.vf1 < (1ll << 31);
}

cudaError_t launch_piv2d_strip(const Piv2dArgs& a, int alg, cudaStream_t s, std::string& err) {
  if (a.ia_end <= a.ia_begin) return cudaSuccess;
  const long long n_ia = a.ia_end - a.ia_begin;
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = device_sm_count(dev);
  // A pass whose IAs all run at once, one to a block, takes two warps to an IA:
  // the kernel is one IA's latency then.  Past that the pairs start a second
  // wave, strips of four do not.  Measured, strips of four and pairs: kernel, 225 IAs
  // 20.9 and 18.6 us, 256 IAs (interSize 32, margin 10) 36 and 27 us (before the rows
  // loaded in batches; now 17 and 23 as pairs); whole call, 484 IAs 63 and 73 us,
  // 1024 IAs 64 and 95 (up to 441 IAs 63 either way: there the call's host work
  // hides the kernel).  A block's shared memory is within bounds for all that
  // piv2d_strip_ok lets through (80,896 bytes at most).
  const int wpi = n_ia <= (long long)STRIP_BLOCKS * sms ? 2 : 1;
  StripCfg c = strip_cfg(a, wpi == 2 ? 1 : 4, wpi);
  c.v2_0 = (int)(a.ia_begin / a.vf1);
  return alg == ALG_FFTCC ? strip_dt<ALG_FFTCC>(a, c, s, err) : strip_dt<ALG_NSQECC>(a, c, s, err);
}

}  // namespace mqp
