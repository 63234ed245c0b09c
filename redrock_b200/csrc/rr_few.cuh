// Scan of a few targets: chi2(z), coefficients and penalty of single targets
// against every redshift of a template, for batches (or the last targets of
// a batch) too small to fill the 32 lanes of a block of the fused scan, and
// for templates with a bounded solve (NNLS / BVLS) at any batch size.
//
// The fused scan (rr_fused.cuh) puts one target on each lane, so a block
// costs the same with 1 target as with 32.  Here the lanes split the pixels.
// A step is 96 pixels in 32 groups of three; a (target, z) is summed by two
// half-warps (16 lanes each, one group per lane), every lane keeping the Gram
// matrix and y of its pixels in FP64 registers, and at the end 32 partial sums
// are added in a fixed tree.  The order of the sums depends on the pixel grid
// alone, never on how many targets there are or which CTA takes them.
//
// CTA = 8 warps = 8 (target, z): 8 redshifts of one target, or 4 of two.  Warp
// w takes groups 16 (w & 1) .. + 15 of slot w >> 1; its lane 2 g + sub takes
// group g of (target, z) `sub` of the slot.  A step's packed rows (9 KB per
// target) and basis windows (106 rows per redshift) come by bulk copies into
// one of two stages; a stage is refilled as soon as its barrier is passed, so
// two steps are in flight.
//
// Shared-memory reads bound the sweep: a 16-byte read costs a warp four cycles
// when all lanes differ and two when neighbouring lanes share the address (far
// ones that do are not merged), an 8-byte read two and one.  Hence the
// neighbours: two targets of one redshift share every basis read, two
// redshifts of one target every packed-row read.  Per warp and step at 10
// bases, against 263 FP64 issue cycles per SM: 65 x 4 + 36 = 296 cycles for
// one target, 65 x 2 + 36 x 2 = 202 for two.  Three pixels per lane: a basis row
// read serves all three (13 rows instead of 33), and the lanes' reads at a
// stride of three rows of 10 (or 2 or 6) doubles fall into different banks
// without padding inside a window, so a window is one bulk copy.
//
// Measured (DESI grids): 1 target x GALAXY, QSO and 5 STAR templates, from host
// arrays, 20.4 -> 2.0 ms (kernels 19.5 -> 1.1 ms); per target of a pair GALAXY
// 0.53, QSO 0.23, STAR 0.04 ms (0.92, 0.40, 0.34 with a whole warp per (target,
// z) and no sharing); 37 targets, 32 of them fused, 41.8 -> 26.0 ms.  A 5-vector
// NMF template of 3311 redshifts, against the plain chain: 1 target 2.3 -> 1.5
// ms, 7 targets 15.4 -> 5.2, 32 69 -> 21, 100 218 -> 64, 256 559 -> 159.  The FP64
// pipe is 42 % busy on GALAXY with one target and 49 % with two: the warps wait
// for shared-memory reads that 255 registers leave no room to start earlier
// (NMF: L1 73 %, FP64 36 %).
#pragma once
#include <cmath>
#include <cstring>

#include "rr_common.cuh"
#include "rr_lsq_dev.cuh"
#include "rr_solve_dev.cuh"

namespace rr {

constexpr int kFewWarps = 8;
constexpr int kFewThreads = kFewWarps * 32;
constexpr int kFewSlots = kFewWarps / 2;  // two half-warp pairs share a slot's two (target, z)
constexpr int kFewTile = 8;    // (target, z) per tile
constexpr int kFewW = 3;       // pixels per lane and step
constexpr int kFewPix = 32 * kFewW;
constexpr int kFewWin = kFewPix + 2 * kHalfBand;        // basis rows per window
constexpr int kFewRowDoubles = kFewPix * RR_RW;         // packed rows of one step
// distance of the two targets' rows in a stage: the 8 lanes of each in a
// half-warp's 8-byte read take different banks
constexpr int kFewRowStride = kFewRowDoubles + 8;
constexpr int kFewStages = 2;
static_assert(RR_CHUNK % kFewW == 0, "a lane's pixels lie all inside or all outside a segment");

// doubles between two windows of rows of S doubles: neighbouring lanes, three
// rows and one window apart, take different banks
__host__ __device__ constexpr int few_window(int S) {
  int w = kFewWin * S;
  while (w % 16 != (S % 4 == 2 ? 8 : 2)) ++w;
  return w;
}
__host__ __device__ constexpr int few_stage(int S) {
  const int one = kFewRowDoubles + 8 * few_window(S);
  const int two = 2 * kFewRowStride + 4 * few_window(S);
  return ((one > two ? one : two) + 1) & ~1;
}

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

// What a tile covers
struct FewTile {
  const double* lrows;  // packed rows of its first target
  int64_t row_doubles;  // to the next target's
  int tgt;              // first target
  int z0;
  int nz;               // redshifts
  bool two;             // two targets
};

// lane 0 of every warp: start the copies of step i into stage s (thread 0 the
// targets' rows and the barrier's byte count, warp w the window of redshift
// z0 + w)
template <int S>
__device__ __forceinline__ void few_issue(const FewParams& p, const rr_scan_template& tm,
                                          const FewTile& tl, int warp, int i, const FewStep& at,
                                          int s, uint64_t* full) {
  const uint32_t tb = (uint32_t)(at.pixels(p) + 2 * kHalfBand) * S * sizeof(double);
  double* st = rr_few_smem + s * few_stage(S);
  const int rows = tl.two ? 2 * kFewRowStride : kFewRowDoubles;
  if (warp == 0) {
    const uint32_t rb = kFewRowDoubles * sizeof(double);
    mbar_arrive_expect_tx(&full[s], (tl.two ? 2 : 1) * rb + tl.nz * tb);
    bulk_g2s(st, tl.lrows + (int64_t)i * kFewRowDoubles, rb, &full[s]);
    if (tl.two)
      bulk_g2s(st + kFewRowStride, tl.lrows + tl.row_doubles + (int64_t)i * kFewRowDoubles, rb,
               &full[s]);
  }
  if (warp < tl.nz)
    bulk_g2s(st + rows + warp * few_window(S),
             tm.basis + ((int64_t)(tl.z0 + warp) * tm.pix_stride + p.segs[at.seg].basis_offset +
                         at.p0 - kHalfBand) *
                            S,
             tb, &full[s]);
}

// One sweep over the pixels.  RESID = false: Gram m and right-hand side y of
// the lane's pixels; true: their residual sum (g - Tb'.c)^2 into acc (lanes
// with active set).  Returns false, for the whole CTA, when a copy wait ran
// out.
template <int NB, bool RESID>
__device__ __forceinline__ bool few_sweep(const FewParams& p, const rr_scan_template& tm,
                                          const FewTile& tl, bool active, uint64_t* full,
                                          uint32_t& uses, double (&m)[NB * (NB + 1) / 2],
                                          double (&y)[NB], const double (&c)[NB], double& acc) {
  constexpr int S = (NB + 1) & ~1;  // doubles per basis row
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int group = 16 * (warp & 1) + (lane >> 1);  // of three pixels
  const int zi = tl.two ? warp >> 1 : 2 * (warp >> 1) + (lane & 1);
  const int row0 = (tl.two ? (lane & 1) * kFewRowStride : 0) + group;
  const int win0 = (tl.two ? 2 * kFewRowStride : kFewRowDoubles) + zi * few_window(S) +
                   group * kFewW * S;
  FewStep ahead, at;
  for (int i = 0; i < kFewStages && i < p.nstep; ++i) {
    if (lane == 0) few_issue<S>(p, tm, tl, warp, i, ahead, i, full);
    ahead.next(p);
  }
  int s = 0;
  for (int i = 0; i < p.nstep; ++i) {
    const bool ok = mbar_wait(&full[s], (uses >> s) & 1u, p.status);
    uses ^= 1u << s;
    if (ok && active && group * kFewW < at.pixels(p)) {
      const double* rw = rr_few_smem + s * few_stage(S) + row0;
      const double* tr = rr_few_smem + s * few_stage(S) + win0;
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
        // basis row k serves pixel q with band index k - q; back and forth
        // over the pixels, so that every product shares a factor with the
        // one before (see the fused scan)
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
              if (k - q >= 0 && k - q < kBand) tp[q][b] = fma(rk[q], tv.x, tp[q][b]);
#pragma unroll
            for (int qq = 0; qq < kFewW; ++qq) {
              const int q = kFewW - 1 - qq;
              if (k - q >= 0 && k - q < kBand) tp[q][b + 1] = fma(rk[q], tv.y, tp[q][b + 1]);
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
      if (threadIdx.x == 0 && i + 1 < p.nstep)
        mbar_wait(&full[s ^ 1], (uses >> (s ^ 1)) & 1u, p.status);
      return false;
    }
    if (i + kFewStages < p.nstep) {
      if (lane == 0) few_issue<S>(p, tm, tl, warp, i + kFewStages, ahead, s, full);
      ahead.next(p);
    }
    s ^= 1;
  }
  return true;
}
static_assert(kFewStages == 2, "few_sweep alternates between two stages");

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

// Sums of N per-lane values over the 16 lanes of equal lane & 1: each step adds
// lanes `off` apart and leaves each lane half of the values, so a lane ends
// with the sums of values first .. first + N / 16 - 1.
template <int N>
__device__ __forceinline__ void few_scatter_sum(double (&v)[N], int& first) {
  const int lane = threadIdx.x & 31;
  first = 0;
  int n = N;
#pragma unroll
  for (int off = 16; off > 1; off >>= 1) {
    n >>= 1;
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n) {
        const double keep = up ? v[n + i] : v[i];
        const double give = up ? v[i] : v[n + i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
      }
    }
    if (up) first += n;
  }
}

// sums of the two half-warps of every (target, z), and its coefficients
template <int NB>
struct FewShared {
  static constexpr int kSum = NB * (NB + 1) / 2 + NB;
  static constexpr int kPad = (kSum + 15) / 16 * 16;
  double part[2][kFewTile][kPad];
  double c[kFewTile][NB];
  int fix[kFewTile];
};

template <int NB, bool BOUNDED>
__device__ bool few_tile(const FewParams& p, const FewBounds& bd, const rr_scan_template& tm,
                         const FewTile& tl, FewShared<NB>& sh, uint64_t* full, uint32_t& uses) {
  constexpr int kTri = NB * (NB + 1) / 2;
  using Sh = FewShared<NB>;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int half = warp & 1;
  // of the lane in the sweep: (target, z) 2 (warp >> 1) + (lane & 1); of the
  // warp in the solve: (target, z) `warp`
  const int mine = 2 * (warp >> 1) + (lane & 1);
  auto in_tile = [&](int e) { return (tl.two ? e >> 1 : e) < tl.nz; };
  {
    double v[Sh::kPad];
    double(&m)[kTri] = *reinterpret_cast<double(*)[kTri]>(v);
    double(&y)[NB] = *reinterpret_cast<double(*)[NB]>(v + kTri);
    double c[NB], acc = 0.0;
#pragma unroll
    for (int i = 0; i < Sh::kPad; ++i) v[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NB; ++i) c[i] = 0.0;
    if (!few_sweep<NB, false>(p, tm, tl, in_tile(mine), full, uses, m, y, c, acc)) return false;
    int first;
    few_scatter_sum<Sh::kPad>(v, first);
#pragma unroll
    for (int i = 0; i < Sh::kPad / 16; ++i) sh.part[half][mine][first + i] = v[i];
  }
  __syncthreads();
  const int z = tl.z0 + (tl.two ? warp >> 1 : warp);
  const int tgt = tl.tgt + (tl.two ? warp & 1 : 0);
  const bool active = in_tile(warp) && p.rows[tgt] >= 0;
  const int64_t o = active ? (int64_t)p.rows[tgt] * tm.nz + z : 0;
  bool fix = false;
  if (active) {
    double m[kTri], y[NB], c[NB];
#pragma unroll
    for (int i = 0; i < kTri; ++i) m[i] = sh.part[0][warp][i] + sh.part[1][warp][i];
#pragma unroll
    for (int i = 0; i < NB; ++i) y[i] = sh.part[0][warp][kTri + i] + sh.part[1][warp][kTri + i];
    const double wsum = p.wsum[tgt];
    double chi2 = kHugeChi2, err = 0.0;
    if constexpr (BOUNDED) {
      // one lane solves (a serial active-set search); chi2 always is the
      // direct residual of a second sweep: a constrained c is no stationary
      // point of f^T W f - c^T y
      if (lane == 0) {
        bool ok = false;
        double cs[NB], lo[NB], hi[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          cs[i] = 0.0;
          lo[i] = bd.lo[i];
          hi[i] = bd.hi[i];
        }
        if (wsum != 0.0) ok = few_bounded<NB>(tm.method, tm.prior, m, y, lo, hi, cs);
#pragma unroll
        for (int i = 0; i < NB; ++i) c[i] = ok ? cs[i] : 0.0;
        fix = ok;
      }
    } else {
      const bool ok = solve_eval<NB>(tm.method, tm.prior, m, y, p.fwf[tgt], wsum, c, chi2, err);
      fix = ok && err > kChi2FixTol;
    }
    if (lane == 0) {
      tm.zchi2[o] = chi2;
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        tm.zcoeff[o * NB + i] = c[i];
        sh.c[warp][i] = c[i];
      }
      if (tm.oii) {
#pragma unroll
        for (int i = 0; i < NB; ++i) s = fma(c[i], tm.oii[i], s);
        // an all-zero-weight target is skipped before the penalty in redrock
        tm.penalty[o] = (wsum != 0.0 && s < 0.0) ? -s : 0.0;
      }
    }
  }
  if (lane == 0) sh.fix[warp] = fix;
  // ill-conditioned fits (and every bounded one): chi2 as the direct
  // weighted residual, as in the fused scan
  if (__syncthreads_or(lane == 0 && fix)) {
    if (!BOUNDED && p.resweep_counter) {
      if (threadIdx.x == 0) atomicAdd(p.resweep_counter, 1);
      if (lane == 0 && fix) atomicAdd(p.resweep_counter + 1, 1);
    }
    double m[kTri], y[NB], c[NB], acc = 0.0;
#pragma unroll
    for (int i = 0; i < NB; ++i) c[i] = sh.fix[mine] ? sh.c[mine][i] : 0.0;
    if (!few_sweep<NB, true>(p, tm, tl, sh.fix[mine] != 0, full, uses, m, y, c, acc)) return false;
#pragma unroll
    for (int off = 16; off > 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane < 2) sh.part[half][mine][0] = acc;
    __syncthreads();
    if (lane == 0 && fix) tm.zchi2[o] = sh.part[0][warp][0] + sh.part[1][warp][0];
  }
  __syncthreads();  // sh is free for the next tile
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
  __shared__ FewShared<NB> sh;
  uint32_t uses = 0;
  const int64_t ntiles = p.tile_start[p.ntemplate];
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    int t = 0;
    while (t + 1 < p.ntemplate && tile >= p.tile_start[t + 1]) ++t;
    int64_t local = tile - p.tile_start[t];
    // pairs of targets, fastest within a group of four redshifts (the tiles
    // that run together share basis windows in L2), then the last target of
    // an odd count with its eight redshifts to a tile
    const int npair = p.count / 2;
    const int64_t paired = (int64_t)npair * ((p.tm[t].nz + 3) / 4);
    FewTile tl;
    tl.two = local < paired;
    if (tl.two) {
      tl.tgt = 2 * (int)(local % npair);
      tl.z0 = (int)(local / npair) * 4;
    } else {
      tl.tgt = p.count - 1;
      tl.z0 = (int)(local - paired) * 8;
    }
    tl.nz = min(tl.two ? 4 : 8, p.tm[t].nz - tl.z0);
    tl.row_doubles = (int64_t)p.nstep * kFewRowDoubles;
    tl.lrows = p.lrows + tl.tgt * tl.row_doubles;
    if (!few_tile<NB, BOUNDED>(p, bd, p.tm[t], tl, sh, full, uses)) break;
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
    const int64_t nz = p.tm[i].nz;
    p.tile_start[i + 1] =
        p.tile_start[i] + (p.count / 2) * ((nz + 3) / 4) + (p.count % 2) * ((nz + 7) / 8);
  }
  const int64_t ntiles = p.tile_start[npick];
  if (ntiles == 0) return RR_OK;
  FewBounds bd;
  for (int i = 0; i < RR_MAX_NBASIS; ++i) {
    bd.lo[i] = -INFINITY;
    bd.hi[i] = INFINITY;
  }
  const size_t smem = (size_t)kFewStages * few_stage((NB + 1) & ~1) * sizeof(double);
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
