// What the pair scans share (rr_pairs.cu, rr_pairs_ws.cu).
#pragma once
#include <cmath>
#include <cstring>

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

static inline int pairs_params(PairsParams& p, const rr_pair_template* tmpl, const rr_pair_segment* segs,
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

}  // namespace rr
