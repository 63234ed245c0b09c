// Scan of a few targets (rr_few.cuh): the packed rows, the entry points and
// the PCA kernels.
#include "rr_few.cuh"

namespace rr {

// lrows[i][step][k][q][g] = rw of target first + i at pixel p0 + 3 g + q of the
// step, 0 past the segment's padded end.  Reads one 8-byte column of
// the fused scan's lane-fastest rows per target (a 32-byte sector each for
// one target, whole sectors from four targets on): 3 MB for a DESI target
// against the 2 GB of basis the scan then reads.
__global__ void __launch_bounds__(256) pack_few_kernel(const __grid_constant__ FewParams p,
                                                       const double* __restrict__ rw,
                                                       int64_t npix_block, int64_t first,
                                                       double* __restrict__ lrows) {
  int seg = 0;
  int step = blockIdx.x;
  for (; seg < p.nseg; ++seg) {
    const int n = (int)((p.segs[seg].npix_pad + kFewPix - 1) / kFewPix);
    if (step < n) break;
    step -= n;
  }
  const int64_t p0 = (int64_t)step * kFewPix;
  const int64_t npad = p.segs[seg].npix_pad;
  // consecutive threads take consecutive targets, then pixels
  for (int e = threadIdx.x; e < kFewRowDoubles * p.count; e += blockDim.x) {
    const int i = e % p.count;
    const int o = e / p.count;
    const int lane = o & 31;
    const int q = (o >> 5) % kFewW;
    const int k = o / kFewPix;
    const int64_t px = p0 + lane * kFewW + q;
    const int64_t t = first + i;
    double v = 0.0;
    if (px < npad)
      v = rw[(((t / RR_LANES) * npix_block + p.segs[seg].rw_offset + px) * RR_RW + k) * RR_LANES +
             t % RR_LANES];
    lrows[((int64_t)i * gridDim.x + blockIdx.x) * kFewRowDoubles + o] = v;
  }
}

static int few_steps(const rr_scan_targets* tg, int64_t* steps) {
  if (!tg || !tg->segs || tg->nseg < 1 || tg->nseg > 16 || tg->nblock < 1) return RR_EINVAL;
  int64_t n = 0;
  for (int s = 0; s < tg->nseg; ++s) {
    const rr_segment_desc& sd = tg->segs[s];
    if (sd.npix_pad <= 0 || sd.npix_pad % RR_CHUNK || sd.basis_offset < kHalfBand ||
        sd.rw_offset < 0 || sd.rw_offset + sd.npix_pad > tg->npix_block)
      return RR_EINVAL;
    n += (sd.npix_pad + kFewPix - 1) / kFewPix;
  }
  if (n > INT32_MAX) return RR_EINVAL;
  *steps = n;
  return RR_OK;
}

static void few_params(FewParams& p, const rr_scan_targets* tg, int64_t first, int count,
                       int64_t steps) {
  memset(&p, 0, sizeof(p));
  p.nseg = tg->nseg;
  for (int s = 0; s < p.nseg; ++s) p.segs[s] = tg->segs[s];
  p.nstep = (int)steps;
  p.count = count;
  p.fwf = tg->fwf + first;
  p.wsum = tg->wsum + first;
  p.rows = tg->rows + first;
}

int few_pca(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
            int npick, bool overlap, cudaStream_t stream) {
#define RR_FEW_CASE(N) \
  case N:              \
    return launch_few<N, false>(p, templates, pick, npick, overlap, stream);
  switch (nbasis) {
    RR_FEW_CASE(1) RR_FEW_CASE(2) RR_FEW_CASE(3) RR_FEW_CASE(4) RR_FEW_CASE(5)
    RR_FEW_CASE(6) RR_FEW_CASE(7) RR_FEW_CASE(8) RR_FEW_CASE(9) RR_FEW_CASE(10)
    default: return RR_EINVAL;
  }
#undef RR_FEW_CASE
}

}  // namespace rr

using namespace rr;

extern "C" int64_t rr_few_rows_doubles(const rr_scan_targets* targets) {
  int64_t steps = 0;
  if (few_steps(targets, &steps)) return -1;
  return steps * kFewRowDoubles;
}

extern "C" int rr_pack_few(const rr_scan_targets* targets, int64_t first, int32_t count,
                           double* lrows, rr_stream_t stream) {
  int64_t steps = 0;
  int rc = few_steps(targets, &steps);
  if (rc) return rc;
  if (first < 0 || count < 0 || first + count > (int64_t)targets->nblock * RR_LANES)
    return RR_EINVAL;
  if (count == 0) return RR_OK;
  if (!targets->rw || !lrows || !targets->fwf || !targets->wsum || !targets->rows)
    return RR_EINVAL;
  FewParams p;
  few_params(p, targets, first, count, steps);
  pack_few_kernel<<<(unsigned)steps, 256, 0, (cudaStream_t)stream>>>(
      p, targets->rw, targets->npix_block, first, lrows);
  RR_CHECK_LAUNCH();
  return RR_OK;
}

extern "C" int rr_zscan_few(const rr_scan_targets* targets, int64_t first, int32_t count,
                            const double* lrows, const rr_scan_template* templates, int ntemplate,
                            int* resweep, int after_fused, int* status, rr_stream_t stream) {
  int64_t steps = 0;
  int rc = few_steps(targets, &steps);
  if (rc) return rc;
  if (!templates || ntemplate < 1 || ntemplate > RR_MAX_TEMPLATES) return RR_EINVAL;
  if (first < 0 || count < 0 || first + count > (int64_t)targets->nblock * RR_LANES)
    return RR_EINVAL;
  if (count == 0) return RR_OK;
  if (!lrows || !targets->fwf || !targets->wsum || !targets->rows) return RR_EINVAL;
  if (reinterpret_cast<uintptr_t>(lrows) & 15) return RR_EINVAL;
  // launches by nbasis: the largest bases first, then the small ones fill
  // the SMs the last tiles leave idle
  int pick[2][RR_MAX_NBASIS + 1][RR_MAX_TEMPLATES];
  int npick[2][RR_MAX_NBASIS + 1] = {};
  for (int t = 0; t < ntemplate; ++t) {
    const rr_scan_template& tm = templates[t];
    if (tm.nbasis < 1 || tm.nbasis > RR_MAX_NBASIS || tm.nz < 0) return RR_EINVAL;
    if (tm.basis_stride != ((tm.nbasis + 1) & ~1)) return RR_EINVAL;
    if (tm.nz > 0 && (!tm.basis || !tm.zchi2 || !tm.zcoeff)) return RR_EINVAL;
    if (tm.oii && !tm.penalty) return RR_EINVAL;
    if (reinterpret_cast<uintptr_t>(tm.basis) & 15) return RR_EINVAL;
    for (int s = 0; s < targets->nseg; ++s)
      if (targets->segs[s].basis_offset + targets->segs[s].npix_pad + kHalfBand > tm.pix_stride)
        return RR_EINVAL;
    const int b = tm.method == RR_SOLVE_NNLS || tm.method == RR_SOLVE_BVLS;
    pick[b][tm.nbasis][npick[b][tm.nbasis]++] = t;
  }
  FewParams p;
  few_params(p, targets, first, count, steps);
  p.lrows = lrows;
  p.resweep_counter = resweep;
  p.status = status;
  bool overlap = after_fused != 0;
  for (int b = 0; b < 2; ++b)
    for (int nb = RR_MAX_NBASIS; nb >= 1; --nb) {
      const int n = npick[b][nb];
      if (!n) continue;
      cudaStream_t st = (cudaStream_t)stream;
      rc = b == 0    ? few_pca(nb, p, templates, pick[b][nb], n, overlap, st)
           : nb <= 7 ? few_bounded_lo(nb, p, templates, pick[b][nb], n, overlap, st)
                     : few_bounded_hi(nb, p, templates, pick[b][nb], n, overlap, st);
      if (rc) return rc;
      overlap = true;
    }
  return RR_OK;
}
