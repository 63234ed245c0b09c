// Scan of a few targets: chi2(z), coefficients and penalty of single targets
// against every redshift of a template, for batches (or the last targets of
// a batch) too small to fill the 32 lanes of a block of the fused scan, and
// for templates with a bounded solve (NNLS / BVLS) at any batch size.
//
// The fused scan (rr_fused.cuh) puts one target on each lane, so a block
// costs the same with 1 target as with 32.  Here a warp owns one (target, z)
// pair and its lanes split the pixels: lane l takes pixels 3 l .. 3 l + 2 of
// every 96-pixel step, keeps the Gram matrix and y of its pixels in FP64
// registers, and one butterfly per (target, z) adds the 32 partial sums.
// The order of the sums depends on the pixel grid alone, never on how many
// targets there are or which CTA takes them.
//
// CTA = 8 warps = 8 redshifts of one target.  A step's packed rows of the
// target (9 KB, shared by the 8 warps) and the 8 basis windows (106 rows
// each) come by bulk copies into one of two stages; a stage is refilled as
// soon as its barrier is passed, so two steps are in flight.
//
// Why three pixels per lane: a basis row read from shared memory serves the
// three pixels (13 rows for 3 pixels instead of 33), and with rows of 10 (or
// 2 or 6) doubles the lanes' 16-byte reads at a stride of three rows fall
// into different banks without padding, so a window is one bulk copy.  The
// sweep is bound by those shared-memory reads: 332 wavefronts for 263 FP64
// issue cycles per warp and step at 10 bases.  With one target the floor is
// the basis, read once from HBM (2.1 GB for 3311 x 7958 x 10).
//
// Measured (DESI grids, whole call from host arrays): 1 target x GALAXY, QSO
// and 5 STAR templates 20.4 -> 2.2 ms (kernels 19.5 -> 1.3 ms, GALAXY 0.71);
// 37 targets (32 fused, 5 here) 41.6 -> 31.6 ms; 7 targets x a 5-vector NMF
// template of 3311 redshifts 15.4 -> 6.0 ms against the plain chain.  ncu on
// GALAXY: FP64 pipe 42 % busy, the warps wait for shared-memory reads (short
// scoreboard 2.7 of 6.2 cycles per issue) that 255 registers leave no room
// to start earlier.
#pragma once
#include <cmath>
#include <cstring>

#include "rr_common.cuh"
#include "rr_lsq_dev.cuh"
#include "rr_solve_dev.cuh"

namespace rr {

constexpr int kFewWarps = 8;   // redshifts per tile
constexpr int kFewThreads = kFewWarps * 32;
constexpr int kFewW = 3;       // pixels per lane and step
constexpr int kFewPix = 32 * kFewW;
constexpr int kFewWin = kFewPix + 2 * kHalfBand;        // basis rows per window
constexpr int kFewRowDoubles = kFewPix * RR_RW;         // packed rows of one step
constexpr int kFewStages = 2;
static_assert(RR_CHUNK % kFewW == 0, "a lane's pixels lie all inside or all outside a segment");

struct FewParams {
  const double* lrows;   // [count][nstep][12][3][32]
  const double* fwf;     // of the first target
  const double* wsum;
  const int32_t* rows;   // output rows of the targets
  rr_segment_desc segs[16];
  int nseg;
  int count;
  int nstep;
  int ntemplate;
  rr_scan_template tm[RR_MAX_TEMPLATES];
  int64_t tile_start[RR_MAX_TEMPLATES + 1];
  int max_stride;
  int* resweep_counter;
  int* status;
};

extern __shared__ __align__(128) double rr_few_smem[];

// position in the list of steps of a target's segments
struct FewStep {
  int seg = 0;
  int64_t p0 = 0;
  __device__ __forceinline__ int pixels(const FewParams& p) const {
    const int64_t left = p.segs[seg].npix_pad - p0;
    return left < kFewPix ? (int)left : kFewPix;
  }
  __device__ __forceinline__ void next(const FewParams& p) {
    p0 += kFewPix;
    if (p0 >= p.segs[seg].npix_pad) {
      p0 = 0;
      ++seg;
    }
  }
};

// lane 0 of every warp: start the copies of step i into stage s (thread 0
// the target's rows and the barrier's byte count, warp w the window of
// redshift z0 + w)
__device__ __forceinline__ void few_issue(const FewParams& p, const rr_scan_template& tm,
                                          const double* lrows, int z0, int nz, int warp, int i,
                                          const FewStep& at, int s, int stage_doubles,
                                          uint64_t* full) {
  const uint32_t tb = (uint32_t)(at.pixels(p) + 2 * kHalfBand) * tm.basis_stride * sizeof(double);
  double* st = rr_few_smem + s * stage_doubles;
  if (warp == 0) {
    const uint32_t rb = kFewRowDoubles * sizeof(double);
    mbar_arrive_expect_tx(&full[s], rb + nz * tb);
    bulk_g2s(st, lrows + (int64_t)i * kFewRowDoubles, rb, &full[s]);
  }
  if (warp < nz) {
    const double* src = tm.basis + ((int64_t)(z0 + warp) * tm.pix_stride +
                                    p.segs[at.seg].basis_offset + at.p0 - kHalfBand) *
                                       tm.basis_stride;
    bulk_g2s(st + kFewRowDoubles + warp * kFewWin * tm.basis_stride, src, tb, &full[s]);
  }
}

// One sweep over a target's pixels for the warp's redshift.  RESID = false:
// Gram m and right-hand side y; true: the residual sum (g - Tb'.c)^2 into
// acc (warps with active set).  Returns false, for the whole CTA, when a
// copy wait ran out.
template <int NB, bool RESID>
__device__ __forceinline__ bool few_sweep(const FewParams& p, const rr_scan_template& tm,
                                          const double* lrows, int z0, int nz, bool active,
                                          int stage_doubles, uint64_t* full, uint32_t& uses,
                                          double (&m)[NB * (NB + 1) / 2], double (&y)[NB],
                                          const double (&c)[NB], double& acc) {
  constexpr int S = (NB + 1) & ~1;  // doubles per basis row
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  FewStep ahead, at;
  for (int i = 0; i < kFewStages && i < p.nstep; ++i) {
    if (lane == 0) few_issue(p, tm, lrows, z0, nz, warp, i, ahead, i, stage_doubles, full);
    ahead.next(p);
  }
  int s = 0;
  for (int i = 0; i < p.nstep; ++i) {
    const bool ok = mbar_wait(&full[s], (uses >> s) & 1u, p.status);
    uses ^= 1u << s;
    if (ok && active && lane * kFewW < at.pixels(p)) {
      const double* rw = rr_few_smem + s * stage_doubles + lane;
      const double* tr =
          rr_few_smem + s * stage_doubles + kFewRowDoubles + (warp * kFewWin + lane * kFewW) * S;
      if (RESID) {
        double md[kFewW];
#pragma unroll
        for (int q = 0; q < kFewW; ++q) md[q] = 0.0;
#pragma unroll
        for (int k = 0; k < kBand + kFewW - 1; ++k) {
          double tc = 0.0;
#pragma unroll
          for (int b = 0; b < NB; ++b) tc = fma(tr[k * S + b], c[b], tc);
#pragma unroll
          for (int q = 0; q < kFewW; ++q)
            if (k - q >= 0 && k - q < kBand)
              md[q] = fma(rw[((k - q) * kFewW + q) * 32], tc, md[q]);
        }
#pragma unroll
        for (int q = 0; q < kFewW; ++q) {
          const double r = rw[(kBand * kFewW + q) * 32] - md[q];
          acc = fma(r, r, acc);
        }
      } else {
        double tp[kFewW][NB];
#pragma unroll
        for (int q = 0; q < kFewW; ++q)
#pragma unroll
          for (int b = 0; b < NB; ++b) tp[q][b] = 0.0;
        // basis row k serves pixel q with band index k - q
#pragma unroll
        for (int k = 0; k < kBand + kFewW - 1; ++k) {
          double rk[kFewW];
#pragma unroll
          for (int q = 0; q < kFewW; ++q)
            rk[q] = (k - q >= 0 && k - q < kBand) ? rw[((k - q) * kFewW + q) * 32] : 0.0;
#pragma unroll
          for (int b = 0; b + 1 < NB; b += 2) {
            const double2 tv = *reinterpret_cast<const double2*>(tr + k * S + b);
#pragma unroll
            for (int q = 0; q < kFewW; ++q)
              if (k - q >= 0 && k - q < kBand) {
                tp[q][b] = fma(rk[q], tv.x, tp[q][b]);
                tp[q][b + 1] = fma(rk[q], tv.y, tp[q][b + 1]);
              }
          }
          if (NB & 1) {
            const double tv = tr[k * S + NB - 1];
#pragma unroll
            for (int q = 0; q < kFewW; ++q)
              if (k - q >= 0 && k - q < kBand) tp[q][NB - 1] = fma(rk[q], tv, tp[q][NB - 1]);
          }
        }
#pragma unroll
        for (int q = 0; q < kFewW; ++q) {
          const double g = rw[(kBand * kFewW + q) * 32];
#pragma unroll
          for (int b = 0; b < NB; ++b) y[b] = fma(g, tp[q][b], y[b]);
#pragma unroll
          for (int a = 0; a < NB; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b)
              m[a * (a + 1) / 2 + b] = fma(tp[q][a], tp[q][b], m[a * (a + 1) / 2 + b]);
        }
      }
    }
    at.next(p);
    // past this point every warp has read stage s; a wait that ran out
    // anywhere stops the whole CTA
    if (__syncthreads_or(!ok)) {
      // the copies still in flight land before the CTA leaves
      if (threadIdx.x == 0 && i + 1 < p.nstep) mbar_wait(&full[s ^ 1], (uses >> (s ^ 1)) & 1u, p.status);
      return false;
    }
    if (i + kFewStages < p.nstep) {
      if (lane == 0)
        few_issue(p, tm, lrows, z0, nz, warp, i + kFewStages, ahead, s, stage_doubles, full);
      ahead.next(p);
    }
    s ^= 1;
  }
  return true;
}
static_assert(kFewStages == 2, "few_sweep alternates between two stages");

__device__ __forceinline__ double few_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// NNLS / BVLS of the full symmetric M + prior against y, as the plain
// chain's bounded solves (unbounded BVLS: the scan has no bounds argument)
template <int NB>
__device__ __noinline__ bool few_bounded(int method, const double* __restrict__ prior,
                                         const double (&m)[NB * (NB + 1) / 2],
                                         const double (&y)[NB], const double (&lo)[NB],
                                         const double (&hi)[NB], double (&c)[NB]) {
  double full[NB][NB], b[NB];
  for (int i = 0; i < NB; ++i) {
    b[i] = y[i];
    for (int j = 0; j <= i; ++j) {
      double v = m[i * (i + 1) / 2 + j];
      if (prior) v += prior[i * NB + j];
      full[i][j] = full[j][i] = v;
    }
  }
  if (method == RR_SOLVE_NNLS) return nnls_solve<NB>(full, b, c);
  return bvls_solve<NB>(full, b, lo, hi, c);
}

struct FewBounds {
  double lo[RR_MAX_NBASIS];
  double hi[RR_MAX_NBASIS];
};

// One (target, 8 redshifts) tile.
template <int NB, bool BOUNDED>
__device__ bool few_tile(const FewParams& p, const FewBounds& bd, const rr_scan_template& tm,
                         int tgt, int z0, int stage_doubles, uint64_t* full, uint32_t& uses) {
  constexpr int kTri = NB * (NB + 1) / 2;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nz = min(kFewWarps, tm.nz - z0);
  const int z = z0 + warp;
  const double* lrows = p.lrows + (int64_t)tgt * p.nstep * kFewRowDoubles;
  const int32_t row = p.rows[tgt];
  const bool active = warp < nz && row >= 0;
  double m[kTri], y[NB], c[NB], acc = 0.0;
#pragma unroll
  for (int i = 0; i < kTri; ++i) m[i] = 0.0;
#pragma unroll
  for (int i = 0; i < NB; ++i) y[i] = 0.0;
  if (!few_sweep<NB, false>(p, tm, lrows, z0, nz, active, stage_doubles, full, uses, m, y, c, acc))
    return false;
  bool fix = false;
  if (active) {
#pragma unroll
    for (int i = 0; i < kTri; ++i) m[i] = few_sum(m[i]);
#pragma unroll
    for (int i = 0; i < NB; ++i) y[i] = few_sum(y[i]);
    const double wsum = p.wsum[tgt];
    double chi2 = kHugeChi2, err = 0.0;
    if constexpr (BOUNDED) {
      // one lane solves (a serial active-set search); chi2 always is the
      // direct residual of a second sweep: a constrained c is no stationary
      // point of f^T W f - c^T y
      int ok = 0;
      double cs[NB];
#pragma unroll
      for (int i = 0; i < NB; ++i) cs[i] = 0.0;
      if (lane == 0 && wsum != 0.0) {
        double ms[kTri], ys[NB], lo[NB], hi[NB];
#pragma unroll
        for (int i = 0; i < kTri; ++i) ms[i] = m[i];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          ys[i] = y[i];
          lo[i] = bd.lo[i];
          hi[i] = bd.hi[i];
        }
        ok = few_bounded<NB>(tm.method, tm.prior, ms, ys, lo, hi, cs) ? 1 : 0;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const double v = __shfl_sync(0xffffffffu, cs[i], 0);
        c[i] = ok ? v : 0.0;
      }
      fix = ok != 0;
    } else {
      const bool ok = solve_eval<NB>(tm.method, tm.prior, m, y, p.fwf[tgt], wsum, c, chi2, err);
      fix = ok && err > kChi2FixTol;
    }
    if (lane == 0) {
      const int64_t o = (int64_t)row * tm.nz + z;
      tm.zchi2[o] = chi2;
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < NB; ++i) tm.zcoeff[o * NB + i] = c[i];
      if (tm.oii) {
#pragma unroll
        for (int i = 0; i < NB; ++i) s = fma(c[i], tm.oii[i], s);
        // an all-zero-weight target is skipped before the penalty in redrock
        tm.penalty[o] = (wsum != 0.0 && s < 0.0) ? -s : 0.0;
      }
    }
  }
  // ill-conditioned fits (and every bounded one): chi2 as the direct
  // weighted residual, as in the fused scan
  if (__syncthreads_or(fix)) {
    if (!BOUNDED && p.resweep_counter) {
      if (threadIdx.x == 0) atomicAdd(p.resweep_counter, 1);
      if (lane == 0 && fix) atomicAdd(p.resweep_counter + 1, 1);
    }
    acc = 0.0;
    if (!few_sweep<NB, true>(p, tm, lrows, z0, nz, fix, stage_doubles, full, uses, m, y, c, acc))
      return false;
    if (fix) {
      acc = few_sum(acc);
      if (lane == 0) tm.zchi2[(int64_t)row * tm.nz + z] = acc;
    }
  }
  return true;
}

// bases of up to 5 vectors leave registers and shared memory for two CTAs
template <int NB, bool BOUNDED>
__global__ void __launch_bounds__(kFewThreads, (NB <= 5 ? 2 : 1))
    zscan_few_kernel(const __grid_constant__ FewParams p, const __grid_constant__ FewBounds bd) {
  __shared__ __align__(8) uint64_t full[kFewStages];
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFewStages; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int stage_doubles = kFewRowDoubles + kFewWarps * kFewWin * ((NB + 1) & ~1);
  uint32_t uses = 0;
  const int64_t ntiles = p.tile_start[p.ntemplate];
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    int t = 0;
    while (t + 1 < p.ntemplate && tile >= p.tile_start[t + 1]) ++t;
    const int64_t local = tile - p.tile_start[t];
    // targets fastest: the tiles that run together share basis windows in L2
    const int tgt = (int)(local % p.count);
    const int z0 = (int)(local / p.count) * kFewWarps;
    if (!few_tile<NB, BOUNDED>(p, bd, p.tm[t], tgt, z0, stage_doubles, full, uses)) break;
  }
  // stream order for whatever follows (see rr_fused.cuh)
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int NB, bool BOUNDED>
int launch_few(FewParams& p, const rr_scan_template* templates, const int* pick, int npick,
               bool overlap, cudaStream_t stream) {
  p.ntemplate = npick;
  p.tile_start[0] = 0;
  for (int i = 0; i < npick; ++i) {
    p.tm[i] = templates[pick[i]];
    const int64_t zt = (p.tm[i].nz + kFewWarps - 1) / kFewWarps;
    p.tile_start[i + 1] = p.tile_start[i] + zt * p.count;
  }
  const int64_t ntiles = p.tile_start[npick];
  if (ntiles == 0) return RR_OK;
  FewBounds bd;
  for (int i = 0; i < RR_MAX_NBASIS; ++i) {
    bd.lo[i] = -INFINITY;
    bd.hi[i] = INFINITY;
  }
  const size_t smem = (size_t)kFewStages *
                      (kFewRowDoubles + kFewWarps * kFewWin * ((NB + 1) & ~1)) * sizeof(double);
  RR_CUDA_TRY(cudaFuncSetAttribute(zscan_few_kernel<NB, BOUNDED>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0, per_sm = 1;
  RR_CUDA_TRY(cudaGetDevice(&dev));
  RR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  RR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, zscan_few_kernel<NB, BOUNDED>, kFewThreads, smem));
  if (per_sm < 1) per_sm = 1;
  const int64_t slots = (int64_t)nsm * per_sm;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(ntiles < slots ? ntiles : slots));
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  RR_CUDA_TRY(cudaLaunchKernelEx(&cfg, zscan_few_kernel<NB, BOUNDED>, p, bd));
  RR_CHECK_LAUNCH();
  return RR_OK;
}

// one entry per translation unit: PCA and bounded solves, nbasis 1..10
int few_pca(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
            int npick, bool overlap, cudaStream_t stream);
int few_bounded_lo(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
                   int npick, bool overlap, cudaStream_t stream);
int few_bounded_hi(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
                   int npick, bool overlap, cudaStream_t stream);

}  // namespace rr
