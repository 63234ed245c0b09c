// Pair scan: chi2, coefficients and [OII] penalty for an arbitrary list of
// (target, redshift) pairs, with the template rebinned on the fly.
//
// This is the batched form of redrock's fine-grid refinement (fitz.py:133-
// 395: for every coarse minimum, rebin_template + transmission_Lyman +
// calc_zchi2_batch on a 15-point grid, then a single-z fit at the parabola
// minimum).  Each target's fine redshifts are its own, so no basis is shared
// between targets: every CTA owns one pair, rebins the template for that
// redshift into shared memory chunk by chunk (the same bit-exact rebin and
// IGM code as the basis builder), and accumulates the banded R.T, the
// weighted Gram matrix and y in FP64 exactly as the fused scan does.
//
//   rows[t][p][12]: sqrt(w) R band rows and sqrt(w) f of target t, pixel p
//                   (rr_pack_rows; segment s starts at segs[s].rw_offset)
//
// Per chunk of 246 output pixels, thread i computes basis row c0 - 5 + i
// (256 rows = chunk + halo), then thread i < 246 forms Tb' for pixel c0 + i
// from shared rows i..i+10.  Template samples covering the chunk are staged
// in shared memory first, so the per-pixel search for the first sample
// beyond a bin edge runs on shared memory.  rr_zscan_pairs_ws (below) does
// the same in rounds through a workspace.
#include <cstring>

#include "rr_build.cuh"
#include "rr_lsq_dev.cuh"
#include "rr_rebin_dev.cuh"
#include "rr_solve_dev.cuh"

namespace rr {

constexpr int kPairThreads = 256;
constexpr int kPairChunk = kPairThreads - 2 * kHalfBand;  // output pixels per chunk
constexpr int kPairMaxSeg = 16;
constexpr int kPairWin = 1536;  // template samples staged per chunk

struct PairsParams {
  rr_pair_template tm;
  rr_pair_segment segs[kPairMaxSeg];
  int nseg;
  const double* rows;
  const double* fwf;
  const double* wsum;
  int64_t npix_row;
  const int32_t* pair_target;
  const double* pair_z;
  int64_t npairs;
  double* chi2;
  double* coeff;
  double* penalty;
  // gradient mode (rr_zscan_pairs_grad)
  double* dchi2_dz;     // [npairs]
  double* d2chi2_dz2;   // [npairs]
  double* dchi2_dflux;  // [npairs][npix_row] or NULL
  double* dpen_dz;      // [npairs] d penalty / dz or NULL
  const double* sw;     // [ntarget][npix_row] sqrt(w), needed for dchi2_dflux
  int* status;
  // RR_SOLVE_BVLS bounds (+-inf when the caller gives none); read in place
  // by the solver, like the plain chain's
  double lo[RR_MAX_NBASIS];
  double hi[RR_MAX_NBASIS];
};

// odd row stride (doubles) of the shared basis rows: conflict-free 64-bit
// reads by consecutive threads
template <int NB>
constexpr int pair_stride() { return (NB & 1) ? NB : NB + 1; }

template <int NB>
struct PairSmem {
  double t[kPairThreads * pair_stride<NB>()];  // basis rows of the chunk + halo
  double dt[kPairThreads * pair_stride<NB>()]; // their z derivatives (gradient mode)
  double xs[kPairWin];                          // staged template wavelengths
  double ys[NB * kPairWin];                     // staged template fluxes
  double red[kPairThreads / 32][NB * (NB + 1) / 2 + NB];
  double c[NB];
  int64_t jlo, jhi, win;
  int fix;
  int bad;
};

// Fill the shared basis rows for output pixels [c0 - 5, c0 + kPairChunk + 5)
// of segment sg at redshift z.  Returns false if a bin fell outside the
// template (never for pairs that pass the host-side range check).
template <int NB, bool DZ>
__device__ bool fill_rows(const PairsParams& p, const rr_pair_segment& sg, int64_t c0, double z,
                          double zp1, bool igm, PairSmem<NB>& sm) {
  constexpr int S = pair_stride<NB>();
  const rr_pair_template& tm = p.tm;
  const int64_t first = c0 - kHalfBand;
  const int64_t last = min(c0 + kPairChunk + kHalfBand, sg.npix);  // exclusive
  // samples needed: from the one before the first edge to the one after
  // the last edge; the two searches (guess from the near-uniform sample
  // spacing, then a short walk: a few dependent loads instead of a binary
  // search's ~16) run in two warps at once
  if (threadIdx.x == 0) {
    const int64_t e0 = max(first, (int64_t)0);
    sm.jlo = max(first_above(tm.x, tm.nx, zp1, sg.edges[e0]) - 2, (int64_t)0);
  } else if (threadIdx.x == 32) {
    sm.jhi = min(first_above(tm.x, tm.nx, zp1, sg.edges[last]) + 2, tm.nx);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int64_t span = sm.jhi - sm.jlo;
    sm.win = (span > 0 && span <= kPairWin) ? span : 0;  // 0: use global arrays
  }
  __syncthreads();
  const int64_t jlo = sm.jlo, win = sm.win;
  for (int64_t i = threadIdx.x; i < win; i += kPairThreads) {
    sm.xs[i] = tm.x[jlo + i];
#pragma unroll
    for (int b = 0; b < NB; ++b) sm.ys[b * kPairWin + i] = tm.y[(int64_t)b * tm.nx + jlo + i];
  }
  __syncthreads();
  bool ok = true;
  const int64_t ip = first + threadIdx.x;
  double* row = sm.t + threadIdx.x * S;
  double* drow = sm.dt + threadIdx.x * S;
  if (ip < 0 || ip >= sg.npix) {
#pragma unroll
    for (int b = 0; b < NB; ++b) row[b] = 0.0;
    if (DZ)
#pragma unroll
      for (int b = 0; b < NB; ++b) drow[b] = 0.0;
  } else {
    double res[kMaxRebinBasis], dres[DZ ? kMaxRebinBasis : 1];
    bool got = false;
    if (win > 0) {
      // rebin on the staged window: the bin must have a sample before and
      // after it inside the window, else fall back to the global arrays
      got = rebin_bin_strided<DZ>(sm.xs, win, sm.ys, kPairWin, NB, zp1, sg.edges[ip],
                                  sg.edges[ip + 1], res, dres);
    }
    if (!got)
      got = rebin_bin_strided<DZ>(tm.x, tm.nx, tm.y, tm.nx, NB, zp1, sg.edges[ip],
                                  sg.edges[ip + 1], res, dres);
    if (!got) {
      ok = false;
#pragma unroll
      for (int b = 0; b < NB; ++b) res[b] = 0.0;
      if (DZ)
#pragma unroll
        for (int b = 0; b < NB; ++b) dres[b] = 0.0;
    }
    if (igm) {
      double dtr = 0.0;
      const double tr = DZ ? transmission_dz(tm.igm_model, z, sg.wave[ip], &dtr)
                           : transmission(tm.igm_model, z, sg.wave[ip]);
      if (DZ)
#pragma unroll
        for (int b = 0; b < NB; ++b) dres[b] = dres[b] * tr + res[b] * dtr;
#pragma unroll
      for (int b = 0; b < NB; ++b) res[b] = dmul(res[b], tr);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) row[b] = res[b];
    if (DZ)
#pragma unroll
      for (int b = 0; b < NB; ++b) drow[b] = dres[b];
  }
  __syncthreads();
  return ok;
}

// Sweep modes over every pixel of the pair's target:
//   kGram:  Gram matrix m and y (forward);
//   kResid: residual sum (g - Tb'.c)^2 into acc[0];
//   kGrad:  residual sum, gradient and curvature accumulators with
//           dTb' = R' dT/dz:  acc[0] = sum res^2, acc[1] = sum res (dTb'.c),
//           acc[2] = sum (dTb'.c)^2, acc[3..3+NB) = u = dTb'^T res,
//           acc[3+NB..3+2NB) = v = Tb'^T (dTb'.c); and dchi2/dflux.
enum SweepMode { kGram = 0, kResid = 1, kGrad = 2 };

template <int NB, int MODE>
__device__ bool pair_sweep(const PairsParams& p, int64_t pr, int64_t t, double z,
                           double (&m)[NB * (NB + 1) / 2], double (&y)[NB], const double* c,
                           double* acc, PairSmem<NB>& sm) {
  constexpr int S = pair_stride<NB>();
  constexpr bool DZ = MODE == kGrad;
  const double zp1 = dadd(1.0, z);
  bool ok = true;
  for (int s = 0; s < p.nseg; ++s) {
    const rr_pair_segment& sg = p.segs[s];
    // redrock skips the IGM product when no redshift puts the grid's bluest
    // pixel below Lyman-alpha (igm.py:396-401); the transmission is exactly
    // 1 there anyway
    const bool igm = p.tm.igm_model != RR_IGM_NONE && !(ddiv(sg.wave_min, zp1) > kLyA);
    for (int64_t c0 = 0; c0 < sg.npix; c0 += kPairChunk) {
      ok = fill_rows<NB, DZ>(p, sg, c0, z, zp1, igm, sm) && ok;
      const int64_t ip = c0 + threadIdx.x;
      if (threadIdx.x < kPairChunk && ip < sg.npix) {
        const int64_t prow = (t * p.npix_row) + sg.row_offset + ip;
        const double* rr = p.rows + prow * RR_RW;
        double r[kBand];
#pragma unroll
        for (int k = 0; k < kBand; ++k) r[k] = rr[k];
        const double g = rr[kBand];
        double tb[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) tb[b] = 0.0;
#pragma unroll
        for (int k = 0; k < kBand; ++k) {
          const double* trow = sm.t + (threadIdx.x + k) * S;
#pragma unroll
          for (int b = 0; b < NB; ++b) tb[b] = fma(r[k], trow[b], tb[b]);
        }
        if (MODE == kGram) {
#pragma unroll
          for (int b = 0; b < NB; ++b) y[b] = fma(g, tb[b], y[b]);
#pragma unroll
          for (int a = 0; a < NB; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b)
              m[a * (a + 1) / 2 + b] = fma(tb[a], tb[b], m[a * (a + 1) / 2 + b]);
        } else {
          double model = 0.0;
#pragma unroll
          for (int b = 0; b < NB; ++b) model = fma(tb[b], c[b], model);
          const double res = g - model;
          acc[0] = fma(res, res, acc[0]);
          if (MODE == kGrad) {
            double db[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) db[b] = 0.0;
#pragma unroll
            for (int k = 0; k < kBand; ++k) {
              const double* drow = sm.dt + (threadIdx.x + k) * S;
#pragma unroll
              for (int b = 0; b < NB; ++b) db[b] = fma(r[k], drow[b], db[b]);
            }
            double dm = 0.0;
#pragma unroll
            for (int b = 0; b < NB; ++b) dm = fma(db[b], c[b], dm);
            acc[1] = fma(res, dm, acc[1]);
            acc[2] = fma(dm, dm, acc[2]);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              acc[3 + b] = fma(db[b], res, acc[3 + b]);
              acc[3 + NB + b] = fma(tb[b], dm, acc[3 + NB + b]);
            }
            // d chi2 / d f_p = 2 w_p r_p = 2 sqrt(w_p) * (sqrt(w_p) r_p)
            if (p.dchi2_dflux)
              p.dchi2_dflux[pr * p.npix_row + sg.row_offset + ip] =
                  2.0 * p.sw[prow] * res;
          }
        }
      }
      __syncthreads();  // rows of this chunk fully consumed
    }
  }
  return ok;
}

// Deterministic block sum of v[0..n) (fixed shuffle tree, then warps in order).
template <int NB>
__device__ void block_sum(double* v, int n, PairSmem<NB>& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = 0; e < n; ++e) {
    double x = v[e];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    if (lane == 0) sm.red[warp][e] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int e = 0; e < n; ++e) {
      double x = sm.red[0][e];
      for (int w = 1; w < kPairThreads / 32; ++w) x += sm.red[w][e];
      v[e] = x;
    }
  }
  __syncthreads();
}

// the plain chain's bounded solves (plain_lsq_kernel) on one pair's
// packed M and y: the full symmetric M + prior, then NNLS or BVLS
template <int NB>
__device__ __noinline__ bool bounded_solve(const PairsParams& p, const double (&mm)[NB * (NB + 1) / 2],
                                           const double (&yy)[NB], double (&c)[NB]) {
  double full[NB][NB], b[NB];
  for (int i = 0; i < NB; ++i) {
    b[i] = yy[i];
    for (int j = 0; j <= i; ++j) {
      double v = mm[i * (i + 1) / 2 + j];
      if (p.tm.prior) v += p.tm.prior[i * NB + j];
      full[i][j] = full[j][i] = v;
    }
  }
  bool ok;
  if (p.tm.method == RR_SOLVE_NNLS)
    ok = nnls_solve<NB>(full, b, c);
  else if (p.tm.method == RR_SOLVE_BVLS)
    ok = bvls_solve<NB>(full, b, p.lo, p.hi, c);
  else
    ok = false;
  if (!ok)
    for (int i = 0; i < NB; ++i) c[i] = 0.0;
  return ok;
}

template <int NB, bool GRAD>
__global__ void __launch_bounds__(kPairThreads, (NB <= 5 ? 2 : 1)) zscan_pairs_kernel(const __grid_constant__ PairsParams p) {
  extern __shared__ __align__(16) unsigned char pair_smem_raw[];
  PairSmem<NB>& sm = *reinterpret_cast<PairSmem<NB>*>(pair_smem_raw);
  constexpr int kTri = NB * (NB + 1) / 2;
  constexpr int kAcc = 3 + 2 * NB;
  for (int64_t pr = blockIdx.x; pr < p.npairs; pr += gridDim.x) {
    const int64_t t = p.pair_target[pr];
    const double z = p.pair_z[pr];
    double m[kTri + NB];
    double(&mm)[kTri] = *reinterpret_cast<double(*)[kTri]>(m);
    double(&yy)[NB] = *reinterpret_cast<double(*)[NB]>(m + kTri);
#pragma unroll
    for (int i = 0; i < kTri + NB; ++i) m[i] = 0.0;
    double acc[kAcc];
#pragma unroll
    for (int i = 0; i < kAcc; ++i) acc[i] = 0.0;
    bool ok = pair_sweep<NB, kGram>(p, pr, t, z, mm, yy, nullptr, acc, sm);
    if (!__syncthreads_and(ok)) {
      if (threadIdx.x == 0) {
        set_status(p.status, RR_ERANGE);
        p.chi2[pr] = nan("");
        for (int b = 0; b < NB; ++b) p.coeff[pr * NB + b] = nan("");
        if (p.penalty) p.penalty[pr] = nan("");
        if (GRAD) {
          p.dchi2_dz[pr] = nan("");
          p.d2chi2_dz2[pr] = nan("");
          if (p.dpen_dz) p.dpen_dz[pr] = nan("");
        }
      }
      continue;
    }
    block_sum<NB>(m, kTri + NB, sm);
    bool solved = false;
    if (threadIdx.x == 0) {
      double c[NB], chi2 = 0.0, err = 0.0;
      if (GRAD || p.tm.method == RR_SOLVE_PCA) {
        solved = solve_eval<NB>(p.tm.method, p.tm.prior, mm, yy, p.fwf[t], p.wsum[t], c, chi2,
                                err);
        sm.fix = (solved && err > kChi2FixTol) ? 1 : 0;
      } else {
        // NMF / NNLS / BVLS (calc_zchi2_batch's bounded branches): the
        // solver on M + prior and y, then chi2 always as the direct
        // residual (a constrained c is no stationary point of
        // f^T W f - c^T y); a failed solve gives HUGE_CHI2, zero c
        solved = bounded_solve<NB>(p, mm, yy, c);
        chi2 = kHugeChi2;
        sm.fix = solved ? 1 : 0;
      }
      sm.bad = solved ? 0 : 1;
      for (int b = 0; b < NB; ++b) sm.c[b] = c[b];
      p.chi2[pr] = chi2;
      for (int b = 0; b < NB; ++b) p.coeff[pr * NB + b] = c[b];
      if (p.penalty) {
        double s = 0.0;
        if (p.tm.oii)
          for (int b = 0; b < NB; ++b) s = fma(c[b], p.tm.oii[b], s);
        p.penalty[pr] = (p.wsum[t] != 0.0 && s < 0.0) ? -s : 0.0;
      }
    }
    __syncthreads();
    if (GRAD) {
      if (sm.bad) {
        if (threadIdx.x == 0) {
          p.dchi2_dz[pr] = 0.0;
          p.d2chi2_dz2[pr] = 0.0;
          if (p.dpen_dz) p.dpen_dz[pr] = 0.0;
        }
        __syncthreads();
        continue;
      }
      // residual chi2 (exact), gradient and curvature in one more sweep
      pair_sweep<NB, kGrad>(p, pr, t, z, mm, yy, sm.c, acc, sm);
      block_sum<NB>(acc, kAcc, sm);
      if (threadIdx.x == 0) {
        // envelope curvature: 2 sum (dTb'.c)^2 - 2 (u - v)^T (M + P)^-1 (u - v)
        double mp[kTri], uv[NB], x[NB];
#pragma unroll
        for (int i = 0; i < kTri; ++i) mp[i] = mm[i];
        if (p.tm.prior)
#pragma unroll
          for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) mp[i * (i + 1) / 2 + j] += p.tm.prior[i * NB + j];
#pragma unroll
        for (int b = 0; b < NB; ++b) uv[b] = acc[3 + b] - acc[3 + NB + b];
        double q = 0.0;
        const bool xok = ldlt_solve<NB>(mp, uv, x);
        if (xok)
#pragma unroll
          for (int b = 0; b < NB; ++b) q = fma(uv[b], x[b], q);
        p.chi2[pr] = acc[0];
        p.dchi2_dz[pr] = -2.0 * acc[1];
        p.d2chi2_dz2[pr] = 2.0 * acc[2] - 2.0 * q;
        if (p.dpen_dz) {
          // x = dc/dz = (M + P)^-1 (u - v); the penalty -c.oii (when the
          // [OII] model is negative) changes by -x.oii
          double s = 0.0, ds = 0.0;
          if (p.tm.oii)
            for (int b = 0; b < NB; ++b) {
              s = fma(sm.c[b], p.tm.oii[b], s);
              ds = fma(xok ? x[b] : 0.0, p.tm.oii[b], ds);
            }
          p.dpen_dz[pr] = (p.wsum[t] != 0.0 && s < 0.0) ? -ds : 0.0;
        }
      }
      __syncthreads();
      continue;
    }
    if (sm.fix) {
      // ill-conditioned: chi2 as the direct residual sum w (f - Tb c)^2
      acc[0] = 0.0;
      pair_sweep<NB, kResid>(p, pr, t, z, mm, yy, sm.c, acc, sm);
      block_sum<NB>(acc, 1, sm);
      if (threadIdx.x == 0) p.chi2[pr] = acc[0];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// the pair scan with a workspace (rr_zscan_pairs_ws)
// ---------------------------------------------------------------------------
// Without a workspace (zscan_pairs_kernel) a CTA rebins the template chunk by
// chunk between barriers and spends most of its time waiting for loads (FP64
// pipe 12 % busy).  With one, a round of pairs runs as
//   1. build_basis_rows: the template of every pair's redshift, as the basis
//      builder makes it for a template's redshifts, into the workspace;
//   2. pairs_gram_kernel: M and y per pair from bulk-copied chunks of basis
//      and target rows, three chunks in flight across pair boundaries;
//   3. pairs_solve_kernel: one thread per pair;
//   4. pairs_resid_kernel: the direct residual for the pairs that need it.
// Every sum keeps zscan_pairs_kernel's order (thread i of the chunk owns pixel
// c0 + i, the warp tree, then the warps), so the results are the same bits.
//
// The Gram kernel is bound by its shared-memory reads: 55 16-byte reads of
// basis rows (conflict-free at a stride of 80 bytes) and 6 of target rows
// per pixel, 268 wavefronts per warp and chunk for 88 FP64 issue cycles at
// 10 bases.  4800 GALAXY pairs on DESI grids: 25.9 -> 7.1 ms (4.5 ms of it
// the rebin, 2.56 ms the Gram kernel).
constexpr int kPgStages = 3;

struct PairsWsParams {
  rr_pair_segment segs[kPairMaxSeg];
  int64_t basis_off[kPairMaxSeg];  // padded index of a segment's first pixel
  int nseg;
  int nchunk;                      // chunks per pair
  const double* basis;             // [n][pix_stride][S]
  int64_t pix_stride;
  const double* rows;
  int64_t npix_row;
  const int32_t* pair_target;      // of the round's first pair
  int64_t n;
  double* my;                      // [n][kTri + NB]
  const double* coeff;             // residual pass
  const int* fix;                  // residual pass: pairs to sum
  double* chi2;
  int* status;
};

// position in the (pair, segment, chunk) sequence of a CTA
struct PairStep {
  int64_t pr;
  int seg = 0;
  int64_t c0 = 0;
  int64_t t;
  __device__ __forceinline__ void start(const PairsWsParams& p, int64_t pair) {
    pr = pair;
    seg = 0;
    c0 = 0;
    t = pr < p.n ? p.pair_target[pr] : 0;
  }
  __device__ __forceinline__ int pixels(const PairsWsParams& p) const {
    const int64_t left = p.segs[seg].npix - c0;
    return left < kPairChunk ? (int)left : kPairChunk;
  }
  // next chunk; the next pair of the CTA after the last one
  __device__ __forceinline__ void next(const PairsWsParams& p) {
    c0 += kPairChunk;
    if (c0 < p.segs[seg].npix) return;
    c0 = 0;
    if (++seg == p.nseg) start(p, pr + gridDim.x);
  }
};

template <int S>
struct PairStage {
  static constexpr int kT = kPairThreads * S;        // basis rows of a chunk and its halo
  static constexpr int kDoubles = kT + kPairChunk * RR_RW;
};

extern __shared__ __align__(128) double pair_stage_smem[];

template <int S>
__device__ __forceinline__ void pair_issue(const PairsWsParams& p, const PairStep& at, int s,
                                           uint64_t* full) {
  const int n = at.pixels(p);
  const uint32_t tb = (uint32_t)(n + 2 * kHalfBand) * S * sizeof(double);
  const uint32_t rb = (uint32_t)n * RR_RW * sizeof(double);
  double* st = pair_stage_smem + s * PairStage<S>::kDoubles;
  mbar_arrive_expect_tx(&full[s], tb + rb);
  bulk_g2s(st, p.basis + (at.pr * p.pix_stride + p.basis_off[at.seg] + at.c0 - kHalfBand) * S, tb,
           &full[s]);
  bulk_g2s(st + PairStage<S>::kT,
           p.rows + (at.t * p.npix_row + p.segs[at.seg].row_offset + at.c0) * RR_RW, rb, &full[s]);
}

// Tb' of the thread's pixel from its 11 basis rows and its packed row
template <int NB>
__device__ __forceinline__ double pair_tb(const double* st, double (&tb)[NB]) {
  constexpr int S = (NB + 1) & ~1;
  const double2* rr =
      reinterpret_cast<const double2*>(st + PairStage<S>::kT + threadIdx.x * RR_RW);
  double r[RR_RW];
#pragma unroll
  for (int k = 0; k < RR_RW / 2; ++k) {
    const double2 v = rr[k];
    r[2 * k] = v.x;
    r[2 * k + 1] = v.y;
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) tb[b] = 0.0;
#pragma unroll
  for (int k = 0; k < kBand; ++k) {
    const double* trow = st + (threadIdx.x + k) * S;
#pragma unroll
    for (int b = 0; b + 1 < NB; b += 2) {
      const double2 v = *reinterpret_cast<const double2*>(trow + b);
      tb[b] = fma(r[k], v.x, tb[b]);
      tb[b + 1] = fma(r[k], v.y, tb[b + 1]);
    }
    if (NB & 1) tb[NB - 1] = fma(r[k], trow[NB - 1], tb[NB - 1]);
  }
  return r[kBand];
}

// Sums of N per-lane values over a warp: each of the five steps adds lanes
// off apart (the tree of an xor butterfly) and leaves each lane half of the
// values, so a lane ends with N / 32 sums, of values lane_first + i.
template <int N>
__device__ __forceinline__ void warp_scatter_sum(double* v, int& lane_first) {
  const int lane = threadIdx.x & 31;
  lane_first = 0;
  int n = N;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
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
    if (up) lane_first += n;
  }
}

template <int NB>
__global__ void __launch_bounds__(kPairThreads, (NB <= 5 ? 2 : 1))
    pairs_gram_kernel(const __grid_constant__ PairsWsParams p) {
  constexpr int S = (NB + 1) & ~1;
  constexpr int kTri = NB * (NB + 1) / 2;
  constexpr int kSum = kTri + NB;
  constexpr int kPad = (kSum + 31) / 32 * 32;
  __shared__ __align__(8) uint64_t full[kPgStages];
  __shared__ double red[kPairThreads / 32][kPad];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPgStages; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  PairStep ahead;
  ahead.start(p, blockIdx.x);
  if (threadIdx.x == 0)
    for (int i = 0; i < kPgStages && ahead.pr < p.n; ++i) {
      pair_issue<S>(p, ahead, i, full);
      ahead.next(p);
    }
  uint32_t uses = 0;
  int s = 0;
  for (int64_t pr = blockIdx.x; pr < p.n; pr += gridDim.x) {
    double v[kPad];  // M (lower triangle), y, padding
#pragma unroll
    for (int i = 0; i < kPad; ++i) v[i] = 0.0;
    for (int sg = 0; sg < p.nseg; ++sg)
      for (int64_t c0 = 0; c0 < p.segs[sg].npix; c0 += kPairChunk) {
        const int64_t left = p.segs[sg].npix - c0;
        const int n = left < kPairChunk ? (int)left : kPairChunk;
        const bool ok = mbar_wait(&full[s], (uses >> s) & 1u, p.status);
        uses ^= 1u << s;
        if (ok && threadIdx.x < n) {
          double tb[NB];
          const double g = pair_tb<NB>(pair_stage_smem + s * PairStage<S>::kDoubles, tb);
#pragma unroll
          for (int b = 0; b < NB; ++b) v[kTri + b] = fma(g, tb[b], v[kTri + b]);
#pragma unroll
          for (int a = 0; a < NB; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b)
              v[a * (a + 1) / 2 + b] = fma(tb[a], tb[b], v[a * (a + 1) / 2 + b]);
        }
        if (__syncthreads_or(!ok)) {
          // the copies still in flight land before the CTA leaves
          if (threadIdx.x == 0)
            for (int q = 1; q < kPgStages; ++q) {
              const int sq = (s + q) % kPgStages;
              mbar_wait(&full[sq], (uses >> sq) & 1u, nullptr);
            }
          return;
        }
        if (threadIdx.x == 0 && ahead.pr < p.n) {
          pair_issue<S>(p, ahead, s, full);
          ahead.next(p);
        }
        s = s + 1 == kPgStages ? 0 : s + 1;
      }
    int first;
    warp_scatter_sum<kPad>(v, first);
#pragma unroll
    for (int i = 0; i < kPad / 32; ++i) red[warp][first + i] = v[i];
    __syncthreads();
    if (threadIdx.x < kSum) {
      double x = red[0][threadIdx.x];
      for (int w = 1; w < kPairThreads / 32; ++w) x += red[w][threadIdx.x];
      p.my[pr * kSum + threadIdx.x] = x;
    }
    // red is read before the next pair's first chunk barrier, written after it
  }
}

// One thread per pair: the solve, chi2, coefficients and penalty of
// zscan_pairs_kernel; fix marks the pairs whose chi2 is the direct residual.
template <int NB>
__global__ void __launch_bounds__(64) pairs_solve_kernel(const __grid_constant__ PairsParams p,
                                                         const double* __restrict__ my,
                                                         const int* __restrict__ bad, int64_t n,
                                                         int* __restrict__ fix) {
  constexpr int kTri = NB * (NB + 1) / 2;
  const int64_t pr = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (pr >= n) return;
  if (bad[pr]) {
    p.chi2[pr] = nan("");
    for (int b = 0; b < NB; ++b) p.coeff[pr * NB + b] = nan("");
    if (p.penalty) p.penalty[pr] = nan("");
    fix[pr] = 0;
    return;
  }
  const int64_t t = p.pair_target[pr];
  double mm[kTri], yy[NB], c[NB], chi2 = 0.0, err = 0.0;
#pragma unroll
  for (int i = 0; i < kTri; ++i) mm[i] = my[pr * (kTri + NB) + i];
#pragma unroll
  for (int i = 0; i < NB; ++i) yy[i] = my[pr * (kTri + NB) + kTri + i];
  bool solved, again;
  if (p.tm.method == RR_SOLVE_NNLS || p.tm.method == RR_SOLVE_BVLS) {
    solved = bounded_solve<NB>(p, mm, yy, c);
    chi2 = kHugeChi2;
    again = solved;
  } else {
    solved = solve_eval<NB>(p.tm.method, p.tm.prior, mm, yy, p.fwf[t], p.wsum[t], c, chi2, err);
    again = solved && err > kChi2FixTol;
  }
  p.chi2[pr] = chi2;
#pragma unroll
  for (int b = 0; b < NB; ++b) p.coeff[pr * NB + b] = c[b];
  if (p.penalty) {
    double s = 0.0;
    if (p.tm.oii)
#pragma unroll
      for (int b = 0; b < NB; ++b) s = fma(c[b], p.tm.oii[b], s);
    p.penalty[pr] = (p.wsum[t] != 0.0 && s < 0.0) ? -s : 0.0;
  }
  fix[pr] = again ? 1 : 0;
}

// chi2 of the marked pairs as the direct residual sum w (f - Tb c)^2
template <int NB>
__global__ void __launch_bounds__(kPairThreads)
    pairs_resid_kernel(const __grid_constant__ PairsWsParams p) {
  constexpr int S = (NB + 1) & ~1;
  __shared__ double red[kPairThreads / 32];
  for (int64_t pr = blockIdx.x; pr < p.n; pr += gridDim.x) {
    if (!p.fix[pr]) continue;  // the same for the whole CTA
    double c[NB], acc = 0.0;
#pragma unroll
    for (int b = 0; b < NB; ++b) c[b] = p.coeff[pr * NB + b];
    const int64_t t = p.pair_target[pr];
    for (int sg = 0; sg < p.nseg; ++sg)
      for (int64_t c0 = 0; c0 < p.segs[sg].npix; c0 += kPairChunk) {
        const int64_t ip = c0 + threadIdx.x;
        if (threadIdx.x >= kPairChunk || ip >= p.segs[sg].npix) continue;
        const double* rr = p.rows + (t * p.npix_row + p.segs[sg].row_offset + ip) * RR_RW;
        const double* tr =
            p.basis + (pr * p.pix_stride + p.basis_off[sg] + ip - kHalfBand) * S;
        double tb[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) tb[b] = 0.0;
#pragma unroll
        for (int k = 0; k < kBand; ++k)
#pragma unroll
          for (int b = 0; b < NB; ++b) tb[b] = fma(rr[k], tr[k * S + b], tb[b]);
        double model = 0.0;
#pragma unroll
        for (int b = 0; b < NB; ++b) model = fma(tb[b], c[b], model);
        const double res = rr[kBand] - model;
        acc = fma(res, res, acc);
      }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double x = red[0];
      for (int w = 1; w < kPairThreads / 32; ++w) x += red[w];
      p.chi2[pr] = x;
    }
    __syncthreads();
  }
}

// workspace of one round: basis rows, M and y, flags (each 256-byte aligned)
struct PairsWsLayout {
  int64_t pix_stride = 0, per_pair = 0;
  int64_t off[kPairMaxSeg];
  int ngrid = 0;
  int grid_seg[kPairMaxSeg];  // a segment of each distinct grid
};

static PairsWsLayout pairs_ws_layout(const rr_pair_segment* segs, int nseg, int nbasis) {
  PairsWsLayout w;
  int64_t grid_off[kPairMaxSeg];
  for (int s = 0; s < nseg; ++s) {
    int g = 0;
    for (; g < w.ngrid; ++g) {
      const rr_pair_segment& o = segs[w.grid_seg[g]];
      if (o.edges == segs[s].edges && o.wave == segs[s].wave && o.npix == segs[s].npix) break;
    }
    if (g == w.ngrid) {
      w.grid_seg[g] = s;
      grid_off[g] = w.pix_stride + kHalfBand;
      w.pix_stride += segs[s].npix + 2 * kHalfBand;
      ++w.ngrid;
    }
    w.off[s] = grid_off[g];
  }
  const int S = (nbasis + 1) & ~1;
  w.per_pair = (w.pix_stride * S + nbasis * (nbasis + 1) / 2 + nbasis) * (int64_t)sizeof(double) +
               2 * (int64_t)sizeof(int);
  return w;
}

template <int NB>
static int launch_pairs_ws(PairsParams p, const PairsWsLayout& w, unsigned char* ws,
                           int64_t per_round, cudaStream_t st) {
  constexpr int S = (NB + 1) & ~1;
  constexpr int kSum = NB * (NB + 1) / 2 + NB;
  double* basis = reinterpret_cast<double*>(ws);
  double* my = basis + per_round * w.pix_stride * S;
  int* bad = reinterpret_cast<int*>(my + per_round * kSum);
  int* fix = bad + per_round;
  PairsWsParams q;
  memset(&q, 0, sizeof(q));
  q.nseg = p.nseg;
  for (int s = 0; s < p.nseg; ++s) {
    q.segs[s] = p.segs[s];
    q.basis_off[s] = w.off[s];
  }
  q.basis = basis;
  q.pix_stride = w.pix_stride;
  q.rows = p.rows;
  q.npix_row = p.npix_row;
  q.my = my;
  q.fix = fix;
  q.status = p.status;
  const size_t smem = (size_t)kPgStages * PairStage<S>::kDoubles * sizeof(double);
  RR_CUDA_TRY(cudaFuncSetAttribute(pairs_gram_kernel<NB>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0, per_sm = 1;
  RR_CUDA_TRY(cudaGetDevice(&dev));
  RR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  RR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pairs_gram_kernel<NB>,
                                                            kPairThreads, smem));
  const int64_t slots = (int64_t)nsm * (per_sm < 1 ? 1 : per_sm);
  const int64_t total = p.npairs;
  const PairsParams all = p;
  for (int64_t i0 = 0; i0 < total; i0 += per_round) {
    const int64_t n = total - i0 < per_round ? total - i0 : per_round;
    RR_CUDA_TRY(cudaMemsetAsync(bad, 0, (size_t)n * sizeof(int), st));
    BuildGrid bg[kPairMaxSeg];
    for (int g = 0; g < w.ngrid; ++g) {
      const rr_pair_segment& sg = p.segs[w.grid_seg[g]];
      bg[g] = BuildGrid{sg.edges, sg.wave, sg.npix, sg.npix, w.off[w.grid_seg[g]], sg.wave_min, 1};
    }
    int rc = build_basis_rows(p.tm.x, p.tm.nx, p.tm.y, NB, all.pair_z + i0, n, bg, w.ngrid,
                              p.tm.igm_model, w.pix_stride, basis, bad, p.status, st);
    if (rc) return rc;
    p.pair_target = all.pair_target + i0;
    p.chi2 = all.chi2 + i0;
    p.coeff = all.coeff + i0 * NB;
    p.penalty = all.penalty ? all.penalty + i0 : nullptr;
    q.pair_target = p.pair_target;
    q.n = n;
    q.coeff = p.coeff;
    q.chi2 = p.chi2;
    pairs_gram_kernel<NB><<<(unsigned)(n < slots ? n : slots), kPairThreads, smem, st>>>(q);
    RR_CHECK_LAUNCH();
    pairs_solve_kernel<NB><<<(unsigned)((n + 63) / 64), 64, 0, st>>>(p, my, bad, n, fix);
    RR_CHECK_LAUNCH();
    const int64_t rg = n < (int64_t)nsm * 8 ? n : (int64_t)nsm * 8;
    pairs_resid_kernel<NB><<<(unsigned)rg, kPairThreads, 0, st>>>(q);
    RR_CHECK_LAUNCH();
  }
  return RR_OK;
}

// rows[t][p][12] for the pair scan; t = block * 32 + lane of the
// spectrum descriptor, row offset of segment s = segs[s].rw_offset.
__global__ void pack_rows_kernel(const rr_spectrum_desc* __restrict__ specs, int64_t nspec,
                                 const double* __restrict__ rdata, const int32_t* __restrict__ roff,
                                 const double* __restrict__ ivar, const double* __restrict__ flux,
                                 const rr_segment_desc* __restrict__ segs, int64_t npix_row,
                                 double* __restrict__ rows, double* __restrict__ sw_out,
                                 int* status) {
  const int64_t s = blockIdx.y;
  if (s >= nspec) return;
  const rr_spectrum_desc sd = specs[s];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= sd.npix) return;
  const rr_segment_desc seg = segs[sd.segment];
  if (seg.rw_offset + i >= npix_row) { set_status(status, RR_EINVAL); return; }
  double r[kBand];
#pragma unroll
  for (int k = 0; k < kBand; ++k) r[k] = 0.0;
  for (int d = 0; d < sd.ndiag; ++d) {
    const int off = roff[sd.diag_offset + d];
    const int64_t j = i + off;
    if (j < 0 || j >= sd.npix) continue;
    const double v = rdata[sd.data_offset + (int64_t)d * sd.npix + j];
    if (off < -kHalfBand || off > kHalfBand) {
      if (v != 0.0) set_status(status, RR_ENOTSUP);
      continue;
    }
    r[off + kHalfBand] += v;
  }
  const double sw = sqrt(ivar[sd.pix_offset + i]);
  const int64_t t = (int64_t)sd.block * RR_LANES + sd.lane;
  double* o = rows + ((t * npix_row) + seg.rw_offset + i) * RR_RW;
#pragma unroll
  for (int k = 0; k < kBand; ++k) o[k] = sw * r[k];
  o[kBand] = sw * flux[sd.pix_offset + i];
  if (sw_out) sw_out[(t * npix_row) + seg.rw_offset + i] = sw;
}

// f^T W f and sum w per target (spectra grouped by target, fixed order)
__global__ void pack_row_sums_kernel(const rr_spectrum_desc* __restrict__ specs,
                                     const int64_t* __restrict__ first, int64_t ntarget,
                                     const double* __restrict__ ivar,
                                     const double* __restrict__ flux, double* __restrict__ fwf,
                                     double* __restrict__ wsum) {
  const int64_t t = blockIdx.x;
  if (t >= ntarget) return;
  __shared__ double red[2][256];
  double ta = 0.0, tb = 0.0;
  for (int64_t s = first[t]; s < first[t + 1]; ++s) {
    const rr_spectrum_desc sd = specs[s];
    double a = 0.0, b = 0.0;
    for (int64_t i = threadIdx.x; i < sd.npix; i += blockDim.x) {
      const double w = ivar[sd.pix_offset + i];
      const double f = flux[sd.pix_offset + i];
      a += w * f * f;
      b += w;
    }
    red[0][threadIdx.x] = a;
    red[1][threadIdx.x] = b;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
      if (threadIdx.x < h) {
        red[0][threadIdx.x] += red[0][threadIdx.x + h];
        red[1][threadIdx.x] += red[1][threadIdx.x + h];
      }
      __syncthreads();
    }
    ta += red[0][0];
    tb += red[1][0];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    fwf[t] = ta;
    wsum[t] = tb;
  }
}

template <int NB, bool GRAD>
static int launch_pairs(const PairsParams& p, cudaStream_t st) {
  const size_t smem = sizeof(PairSmem<NB>);
  if (cudaFuncSetAttribute(zscan_pairs_kernel<NB, GRAD>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return RR_ECUDA;
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RR_ECUDA;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return RR_ECUDA;
  const int64_t grid = p.npairs < (int64_t)nsm * 4 ? p.npairs : (int64_t)nsm * 4;
  zscan_pairs_kernel<NB, GRAD><<<(unsigned)grid, kPairThreads, smem, st>>>(p);
  if (cudaGetLastError() != cudaSuccess) return RR_ECUDA;
  return RR_OK;
}

}  // namespace rr

using namespace rr;

extern "C" int rr_pack_rows(const rr_spectrum_desc* specs, int64_t nspec,
                            const int64_t* target_first, int64_t ntarget, const double* rdata,
                            const int32_t* roffsets, const double* ivar, const double* flux,
                            const rr_segment_desc* segs, int nseg, int64_t npix_row, double* rows,
                            double* sw, double* fwf, double* wsum, int* status,
                            rr_stream_t stream) {
  if (nspec < 0 || ntarget < 0 || nseg < 1 || npix_row < 1) return RR_EINVAL;
  if (nspec == 0 || ntarget == 0) return RR_OK;
  if (!specs || !target_first || !rdata || !roffsets || !ivar || !flux || !segs || !rows || !fwf ||
      !wsum)
    return RR_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  for (int64_t s0 = 0; s0 < nspec; s0 += 65535) {
    const int64_t n = nspec - s0 < 65535 ? nspec - s0 : 65535;
    dim3 block(128);
    dim3 grid((unsigned)((npix_row + block.x - 1) / block.x), (unsigned)n);
    pack_rows_kernel<<<grid, block, 0, st>>>(specs + s0, n, rdata, roffsets, ivar, flux, segs,
                                             npix_row, rows, sw, status);
    if (cudaGetLastError() != cudaSuccess) return RR_ECUDA;
  }
  pack_row_sums_kernel<<<(unsigned)ntarget, 256, 0, st>>>(specs, target_first, ntarget, ivar, flux,
                                                          fwf, wsum);
  if (cudaGetLastError() != cudaSuccess) return RR_ECUDA;
  return RR_OK;
}

static int pairs_params(PairsParams& p, const rr_pair_template* tmpl, const rr_pair_segment* segs,
                        int nseg, const double* rows, const double* fwf, const double* wsum,
                        int64_t npix_row, const int32_t* pair_target, const double* pair_z,
                        int64_t npairs, double* chi2, double* coeff, double* penalty,
                        int* status) {
  if (!tmpl || !segs || nseg < 1 || nseg > kPairMaxSeg || npix_row < 1 || npairs < 0)
    return RR_EINVAL;
  if (npairs > 0 && (!rows || !fwf || !wsum || !pair_target || !pair_z || !chi2 || !coeff))
    return RR_EINVAL;
  if (!tmpl->x || !tmpl->y || tmpl->nx < 2 || tmpl->nbasis < 1 || tmpl->nbasis > RR_MAX_NBASIS)
    return RR_EINVAL;
  if (tmpl->igm_model < RR_IGM_NONE || tmpl->igm_model > RR_IGM_INOUE14) return RR_EINVAL;
  if (tmpl->oii && !penalty) return RR_EINVAL;
  if (tmpl->method < RR_SOLVE_PCA || tmpl->method > RR_SOLVE_BVLS) return RR_EINVAL;
  memset(&p, 0, sizeof(p));
  p.tm = *tmpl;
  for (int i = 0; i < RR_MAX_NBASIS; ++i) {
    p.lo[i] = -INFINITY;
    p.hi[i] = INFINITY;
  }
  if (tmpl->bounds)
    for (int i = 0; i < tmpl->nbasis; ++i) {
      p.lo[i] = tmpl->bounds[i];
      p.hi[i] = tmpl->bounds[tmpl->nbasis + i];
      if (!(p.lo[i] <= p.hi[i])) return RR_EINVAL;
    }
  p.tm.bounds = nullptr;  // host memory: not for the device
  p.nseg = nseg;
  for (int s = 0; s < nseg; ++s) {
    if (segs[s].npix < 1 || !segs[s].edges || !segs[s].wave || segs[s].row_offset < 0 ||
        segs[s].row_offset + segs[s].npix > npix_row)
      return RR_EINVAL;
    p.segs[s] = segs[s];
  }
  p.rows = rows;
  p.fwf = fwf;
  p.wsum = wsum;
  p.npix_row = npix_row;
  p.pair_target = pair_target;
  p.pair_z = pair_z;
  p.npairs = npairs;
  p.chi2 = chi2;
  p.coeff = coeff;
  p.penalty = penalty;
  p.status = status;
  return RR_OK;
}

template <bool GRAD>
static int dispatch_pairs(const PairsParams& p, int nbasis, cudaStream_t st) {
  int rc = upload_igm_tables(st);
  if (rc) return rc;
  switch (nbasis) {
    case 1: return launch_pairs<1, GRAD>(p, st);
    case 2: return launch_pairs<2, GRAD>(p, st);
    case 3: return launch_pairs<3, GRAD>(p, st);
    case 4: return launch_pairs<4, GRAD>(p, st);
    case 5: return launch_pairs<5, GRAD>(p, st);
    case 6: return launch_pairs<6, GRAD>(p, st);
    case 7: return launch_pairs<7, GRAD>(p, st);
    case 8: return launch_pairs<8, GRAD>(p, st);
    case 9: return launch_pairs<9, GRAD>(p, st);
    case 10: return launch_pairs<10, GRAD>(p, st);
    default: return RR_EINVAL;
  }
}

extern "C" int rr_zscan_pairs(const rr_pair_template* tmpl, const rr_pair_segment* segs, int nseg,
                              const double* rows, const double* fwf, const double* wsum,
                              int64_t npix_row, const int32_t* pair_target, const double* pair_z,
                              int64_t npairs, double* chi2, double* coeff, double* penalty,
                              int* status, rr_stream_t stream) {
  PairsParams p;
  int rc = pairs_params(p, tmpl, segs, nseg, rows, fwf, wsum, npix_row, pair_target, pair_z,
                        npairs, chi2, coeff, penalty, status);
  if (rc || npairs == 0) return rc;
  return dispatch_pairs<false>(p, tmpl->nbasis, (cudaStream_t)stream);
}

static bool pair_segments_ok(const rr_pair_segment* segs, int nseg) {
  if (!segs || nseg < 1 || nseg > kPairMaxSeg) return false;
  for (int s = 0; s < nseg; ++s)
    if (segs[s].npix < 1) return false;
  return true;
}

extern "C" size_t rr_zscan_pairs_ws_bytes(const rr_pair_segment* segs, int nseg, int32_t nbasis,
                                          int64_t npairs) {
  if (!pair_segments_ok(segs, nseg) || nbasis < 1 || nbasis > RR_MAX_NBASIS || npairs < 0)
    return SIZE_MAX;
  size_t b = 0;
  if (__builtin_mul_overflow((size_t)pairs_ws_layout(segs, nseg, nbasis).per_pair,
                             (size_t)npairs, &b))
    return SIZE_MAX;
  return b;
}

extern "C" int rr_zscan_pairs_ws(const rr_pair_template* tmpl, const rr_pair_segment* segs,
                                 int nseg, const double* rows, const double* fwf,
                                 const double* wsum, int64_t npix_row, const int32_t* pair_target,
                                 const double* pair_z, int64_t npairs, double* chi2, double* coeff,
                                 double* penalty, void* workspace, size_t workspace_bytes,
                                 int* status, rr_stream_t stream) {
  PairsParams p;
  int rc = pairs_params(p, tmpl, segs, nseg, rows, fwf, wsum, npix_row, pair_target, pair_z,
                        npairs, chi2, coeff, penalty, status);
  if (rc || npairs == 0) return rc;
  if (!workspace || ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(rows)) &
                     15))
    return RR_EINVAL;
  const PairsWsLayout w = pairs_ws_layout(segs, nseg, tmpl->nbasis);
  // an even number of pairs per round keeps the arrays aligned
  int64_t per_round = (int64_t)(workspace_bytes / (size_t)w.per_pair) & ~(int64_t)1;
  if (per_round < 1) return RR_EINVAL;
  // equal rounds, within the builder's grid
  const int64_t most = per_round < 65535 * build_z(false) ? per_round : 65534 * build_z(false);
  const int64_t rounds = (npairs + most - 1) / most;
  per_round = ((npairs + rounds - 1) / rounds + 1) & ~(int64_t)1;
  if (per_round > most) per_round = most;
  cudaStream_t st = (cudaStream_t)stream;
  rc = basis_tables(st);
  if (rc) return rc;
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  switch (tmpl->nbasis) {
    case 1: return launch_pairs_ws<1>(p, w, ws, per_round, st);
    case 2: return launch_pairs_ws<2>(p, w, ws, per_round, st);
    case 3: return launch_pairs_ws<3>(p, w, ws, per_round, st);
    case 4: return launch_pairs_ws<4>(p, w, ws, per_round, st);
    case 5: return launch_pairs_ws<5>(p, w, ws, per_round, st);
    case 6: return launch_pairs_ws<6>(p, w, ws, per_round, st);
    case 7: return launch_pairs_ws<7>(p, w, ws, per_round, st);
    case 8: return launch_pairs_ws<8>(p, w, ws, per_round, st);
    case 9: return launch_pairs_ws<9>(p, w, ws, per_round, st);
    case 10: return launch_pairs_ws<10>(p, w, ws, per_round, st);
    default: return RR_EINVAL;
  }
}

extern "C" int rr_zscan_pairs_grad(const rr_pair_template* tmpl, const rr_pair_segment* segs,
                                   int nseg, const double* rows, const double* sw,
                                   const double* fwf, const double* wsum, int64_t npix_row,
                                   const int32_t* pair_target, const double* pair_z,
                                   int64_t npairs, double* chi2, double* coeff, double* penalty,
                                   double* dchi2_dz, double* d2chi2_dz2, double* dchi2_dflux,
                                   double* dpenalty_dz, int* status, rr_stream_t stream) {
  PairsParams p;
  int rc = pairs_params(p, tmpl, segs, nseg, rows, fwf, wsum, npix_row, pair_target, pair_z,
                        npairs, chi2, coeff, penalty, status);
  if (rc || npairs == 0) return rc;
  if (!dchi2_dz || !d2chi2_dz2 || (dchi2_dflux && !sw)) return RR_EINVAL;
  if (tmpl->method != RR_SOLVE_PCA) return RR_ENOTSUP;
  if (tmpl->prior && dchi2_dflux) return RR_ENOTSUP;
  p.dchi2_dz = dchi2_dz;
  p.d2chi2_dz2 = d2chi2_dz2;
  p.dchi2_dflux = dchi2_dflux;
  p.dpen_dz = dpenalty_dz;
  p.sw = sw;
  return dispatch_pairs<true>(p, tmpl->nbasis, (cudaStream_t)stream);
}
