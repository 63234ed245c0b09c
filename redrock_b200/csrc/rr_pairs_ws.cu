// The pair scan with a workspace (rr_zscan_pairs_ws, rr_zscan_pairs_grad_ws).
#include "rr_build.cuh"
#include "rr_pairs.cuh"

namespace rr {

// ---------------------------------------------------------------------------
// the pair scan with a workspace (rr_zscan_pairs_ws)
// ---------------------------------------------------------------------------
// Without a workspace (zscan_pairs_kernel) a CTA rebins the template chunk by
// chunk between barriers and spends most of its time waiting for loads (FP64
// pipe 12 % busy).  With one, a round of pairs runs as
//   1. build_basis_rows: the template of every pair's redshift, as the basis
//      builder makes it for a template's redshifts, into the workspace;
//   2. pairs_sums_kernel: M and y per pair from bulk-copied chunks of basis
//      and target rows, three chunks in flight across pair boundaries;
//   3. pairs_solve_kernel: one thread per pair;
//   4. pairs_resid_kernel: the direct residual for the pairs that need it, or
//      with gradients pairs_sums_kernel again over T and dT/dz, and
//      pairs_slope_kernel.
// Every sum of 2. to 4. keeps zscan_pairs_kernel's order (thread i of the chunk owns pixel
// c0 + i, the warp tree, then the warps), so the results are the same bits.
//
// The Gram kernel is bound by its shared-memory reads: 55 16-byte reads of
// basis rows (conflict-free at a stride of 80 bytes) and 6 of target rows
// per pixel, 268 wavefronts per warp and chunk for 88 FP64 issue cycles at
// 10 bases (L1 72 % busy, the FP64 pipe 24 %; with gradients 82 and 23 %).
// 4800 GALAXY pairs on DESI grids: 25.9 -> 7.2 ms (4.5 ms of it
// the rebin, 2.6 ms the Gram kernel); 384 GALAXY gradients 2.30 -> 0.92 ms.
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
  const double* coeff;             // residual and gradient passes
  const int* fix;                  // the pairs they take
  double* chi2;
  const double* dbasis;            // gradient pass: dT/dz
  double* acc;                     // its sums [n][3 + 2 NB]
  const double* sw;
  double* dflux;                   // of the round's first pair, or NULL
  int* status;
};

// the CTA's next pair from `pair` on: every one, or those marked in fix
__device__ __forceinline__ int64_t pair_taken(const PairsWsParams& p, int64_t pair) {
  if (p.dbasis)
    while (pair < p.n && !p.fix[pair]) pair += gridDim.x;
  return pair;
}

// position in the (pair, segment, chunk) sequence of a CTA
struct PairStep {
  int64_t pr;
  int seg = 0;
  int64_t c0 = 0;
  int64_t t;
  __device__ __forceinline__ void start(const PairsWsParams& p, int64_t pair) {
    pr = pair_taken(p, pair);
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

template <int S, bool GRAD>
struct PairStage {
  static constexpr int kRows = kPairThreads * S;     // basis rows of a chunk and its halo
  static constexpr int kT = GRAD ? 2 * kRows : kRows;  // and of dT/dz
  static constexpr int kDoubles = kT + kPairChunk * RR_RW;
};

extern __shared__ __align__(128) double pair_stage_smem[];

template <int S, bool GRAD>
__device__ __forceinline__ void pair_issue(const PairsWsParams& p, const PairStep& at, int s,
                                           uint64_t* full) {
  using Stage = PairStage<S, GRAD>;
  const int n = at.pixels(p);
  const uint32_t tb = (uint32_t)(n + 2 * kHalfBand) * S * sizeof(double);
  const uint32_t rb = (uint32_t)n * RR_RW * sizeof(double);
  const int64_t row = (at.pr * p.pix_stride + p.basis_off[at.seg] + at.c0 - kHalfBand) * S;
  double* st = pair_stage_smem + s * Stage::kDoubles;
  mbar_arrive_expect_tx(&full[s], (GRAD ? 2 : 1) * tb + rb);
  bulk_g2s(st, p.basis + row, tb, &full[s]);
  if (GRAD) bulk_g2s(st + Stage::kRows, p.dbasis + row, tb, &full[s]);
  bulk_g2s(st + Stage::kT,
           p.rows + (at.t * p.npix_row + p.segs[at.seg].row_offset + at.c0) * RR_RW, rb, &full[s]);
}

// the thread's packed row
__device__ __forceinline__ void pair_row(const double* rows, double (&r)[RR_RW]) {
  const double2* rr = reinterpret_cast<const double2*>(rows + threadIdx.x * RR_RW);
#pragma unroll
  for (int k = 0; k < RR_RW / 2; ++k) {
    const double2 v = rr[k];
    r[2 * k] = v.x;
    r[2 * k + 1] = v.y;
  }
}

// Tb' of the thread's pixel from 11 basis rows and its packed row
template <int NB>
__device__ __forceinline__ void pair_tb(const double* t, const double (&r)[RR_RW],
                                        double (&tb)[NB]) {
  constexpr int S = (NB + 1) & ~1;
#pragma unroll
  for (int b = 0; b < NB; ++b) tb[b] = 0.0;
#pragma unroll
  for (int k = 0; k < kBand; ++k) {
    const double* trow = t + (threadIdx.x + k) * S;
#pragma unroll
    for (int b = 0; b + 1 < NB; b += 2) {
      const double2 v = *reinterpret_cast<const double2*>(trow + b);
      tb[b] = fma(r[k], v.x, tb[b]);
      tb[b + 1] = fma(r[k], v.y, tb[b + 1]);
    }
    if (NB & 1) tb[NB - 1] = fma(r[k], trow[NB - 1], tb[NB - 1]);
  }
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

// GRAD = false: M and y of every pair.  GRAD = true: for the pairs marked in
// fix, with their coefficients c and dTb' = R' dT/dz, the sums
//   sum res^2, sum res (dTb'.c), sum (dTb'.c)^2, u = dTb'^T res,
//   v = Tb'^T (dTb'.c),
// and dchi2/dflux.
template <int NB, bool GRAD>
__global__ void __launch_bounds__(kPairThreads, (NB <= 5 ? 2 : 1))
    pairs_sums_kernel(const __grid_constant__ PairsWsParams p) {
  constexpr int S = (NB + 1) & ~1;
  using Stage = PairStage<S, GRAD>;
  constexpr int kTri = NB * (NB + 1) / 2;
  constexpr int kSum = GRAD ? 3 + 2 * NB : kTri + NB;
  constexpr int kPad = (kSum + 31) / 32 * 32;
  __shared__ __align__(8) uint64_t full[kPgStages];
  __shared__ double red[kPairThreads / 32][kPad];
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPgStages; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  PairStep ahead;
  ahead.start(p, blockIdx.x);
  int flying = 0;  // chunks issued and not yet waited for (thread 0)
  if (threadIdx.x == 0)
    for (; flying < kPgStages && ahead.pr < p.n; ++flying) {
      pair_issue<S, GRAD>(p, ahead, flying, full);
      ahead.next(p);
    }
  uint32_t uses = 0;
  int s = 0;
  for (int64_t pr = pair_taken(p, blockIdx.x); pr < p.n; pr = pair_taken(p, pr + gridDim.x)) {
    double v[kPad];  // the sums, then padding
#pragma unroll
    for (int i = 0; i < kPad; ++i) v[i] = 0.0;
    double c[GRAD ? NB : 1];
    int64_t t = 0;
    if (GRAD) {
      t = p.pair_target[pr];
#pragma unroll
      for (int b = 0; b < NB; ++b) c[GRAD ? b : 0] = p.coeff[pr * NB + b];
    }
    for (int sg = 0; sg < p.nseg; ++sg)
      for (int64_t c0 = 0; c0 < p.segs[sg].npix; c0 += kPairChunk) {
        const int64_t left = p.segs[sg].npix - c0;
        const int n = left < kPairChunk ? (int)left : kPairChunk;
        const bool ok = mbar_wait(&full[s], (uses >> s) & 1u, p.status);
        uses ^= 1u << s;
        if (ok && threadIdx.x < n) {
          const double* st = pair_stage_smem + s * Stage::kDoubles;
          double r[RR_RW], tb[NB];
          pair_row(st + Stage::kT, r);
          pair_tb<NB>(st, r, tb);
          const double g = r[kBand];
          if constexpr (!GRAD) {
#pragma unroll
            for (int b = 0; b < NB; ++b) v[kTri + b] = fma(g, tb[b], v[kTri + b]);
#pragma unroll
            for (int a = 0; a < NB; ++a)
#pragma unroll
              for (int b = 0; b <= a; ++b)
                v[a * (a + 1) / 2 + b] = fma(tb[a], tb[b], v[a * (a + 1) / 2 + b]);
          } else {
            double model = 0.0, dm = 0.0, db[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) model = fma(tb[b], c[b], model);
            const double res = g - model;
            pair_tb<NB>(st + Stage::kRows, r, db);
#pragma unroll
            for (int b = 0; b < NB; ++b) dm = fma(db[b], c[b], dm);
            v[0] = fma(res, res, v[0]);
            v[1] = fma(res, dm, v[1]);
            v[2] = fma(dm, dm, v[2]);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              v[3 + b] = fma(db[b], res, v[3 + b]);
              v[3 + NB + b] = fma(tb[b], dm, v[3 + NB + b]);
            }
            // d chi2 / d f_p = 2 w_p r_p = 2 sqrt(w_p) (sqrt(w_p) r_p)
            if (p.dflux) {
              const int64_t px = p.segs[sg].row_offset + c0 + threadIdx.x;
              p.dflux[pr * p.npix_row + px] = 2.0 * p.sw[t * p.npix_row + px] * res;
            }
          }
        }
        if (threadIdx.x == 0) --flying;
        if (__syncthreads_or(!ok)) {
          // the copies still in flight land before the CTA leaves
          if (threadIdx.x == 0)
            for (int q = 1; q <= flying; ++q) {
              const int sq = (s + q) % kPgStages;
              mbar_wait(&full[sq], (uses >> sq) & 1u, p.status);
            }
          return;
        }
        if (threadIdx.x == 0 && ahead.pr < p.n) {
          pair_issue<S, GRAD>(p, ahead, s, full);
          ahead.next(p);
          ++flying;
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
      (GRAD ? p.acc : p.my)[pr * kSum + threadIdx.x] = x;
    }
    // red is written again only after the next pair's chunk barriers
  }
}

// One thread per pair: the solve, chi2, coefficients and penalty of
// zscan_pairs_kernel; fix marks the pairs whose chi2 is the direct residual.
// GRAD: the pairs that have a solution are marked for the gradient pass, the
// others get zero derivatives (NaN outside the template range).
template <int NB, bool GRAD>
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
    if (GRAD) {
      p.dchi2_dz[pr] = nan("");
      p.d2chi2_dz2[pr] = nan("");
      if (p.dpen_dz) p.dpen_dz[pr] = nan("");
    }
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
  if (!GRAD && (p.tm.method == RR_SOLVE_NNLS || p.tm.method == RR_SOLVE_BVLS)) {
    solved = bounded_solve<NB>(p, mm, yy, c);
    chi2 = kHugeChi2;
    again = solved;
  } else {
    solved = solve_eval<NB>(p.tm.method, p.tm.prior, mm, yy, p.fwf[t], p.wsum[t], c, chi2, err);
    again = solved && (GRAD || err > kChi2FixTol);
  }
  if (GRAD && !solved) {
    p.dchi2_dz[pr] = 0.0;
    p.d2chi2_dz2[pr] = 0.0;
    if (p.dpen_dz) p.dpen_dz[pr] = 0.0;
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

// One thread per pair: chi2 (the residual sum) and its derivatives from the
// gradient sums; curvature 2 sum (dTb'.c)^2 - 2 (u - v)^T (M + P)^-1 (u - v).
template <int NB>
__global__ void __launch_bounds__(64) pairs_slope_kernel(const __grid_constant__ PairsParams p,
                                                         const double* __restrict__ my,
                                                         const double* __restrict__ sums,
                                                         int64_t n, const int* __restrict__ fix) {
  constexpr int kTri = NB * (NB + 1) / 2;
  const int64_t pr = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (pr >= n || !fix[pr]) return;
  const double* acc = sums + pr * (3 + 2 * NB);
  double mp[kTri], uv[NB], x[NB];
#pragma unroll
  for (int i = 0; i < kTri; ++i) mp[i] = my[pr * (kTri + NB) + i];
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
    // x = dc/dz = (M + P)^-1 (u - v); the penalty -c.oii (when the [OII]
    // model is negative) changes by -x.oii
    double s = 0.0, ds = 0.0;
    if (p.tm.oii)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        s = fma(p.coeff[pr * NB + b], p.tm.oii[b], s);
        ds = fma(xok ? x[b] : 0.0, p.tm.oii[b], ds);
      }
    p.dpen_dz[pr] = (p.wsum[p.pair_target[pr]] != 0.0 && s < 0.0) ? -ds : 0.0;
  }
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

// workspace of one round: basis rows, M and y, flags
struct PairsWsLayout {
  int64_t pix_stride = 0, per_pair = 0;
  int64_t off[kPairMaxSeg];
  int ngrid = 0;
  int grid_seg[kPairMaxSeg];  // a segment of each distinct grid
};

static PairsWsLayout pairs_ws_layout(const rr_pair_segment* segs, int nseg, int nbasis, bool grad) {
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
  const int64_t sums = nbasis * (nbasis + 1) / 2 + nbasis + (grad ? 3 + 2 * nbasis : 0);
  w.per_pair = (w.pix_stride * S * (grad ? 2 : 1) + sums) * (int64_t)sizeof(double) +
               2 * (int64_t)sizeof(int);
  return w;
}

template <int NB, bool GRAD>
static int launch_sums(const PairsWsParams& q, cudaStream_t st) {
  constexpr int S = (NB + 1) & ~1;
  const size_t smem = (size_t)kPgStages * PairStage<S, GRAD>::kDoubles * sizeof(double);
  RR_CUDA_TRY(cudaFuncSetAttribute(pairs_sums_kernel<NB, GRAD>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0, per_sm = 1;
  RR_CUDA_TRY(cudaGetDevice(&dev));
  RR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  RR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pairs_sums_kernel<NB, GRAD>,
                                                            kPairThreads, smem));
  const int64_t slots = (int64_t)nsm * (per_sm < 1 ? 1 : per_sm);
  pairs_sums_kernel<NB, GRAD>
      <<<(unsigned)(q.n < slots ? q.n : slots), kPairThreads, smem, st>>>(q);
  RR_CHECK_LAUNCH();
  return RR_OK;
}

template <int NB, bool GRAD>
static int launch_pairs_ws(PairsParams p, const PairsWsLayout& w, unsigned char* ws,
                           int64_t per_round, cudaStream_t st) {
  constexpr int S = (NB + 1) & ~1;
  constexpr int kSum = NB * (NB + 1) / 2 + NB;
  double* basis = reinterpret_cast<double*>(ws);
  double* dbasis = basis + per_round * w.pix_stride * S;
  double* my = GRAD ? dbasis + per_round * w.pix_stride * S : dbasis;
  double* acc = my + per_round * kSum;
  int* bad = reinterpret_cast<int*>(GRAD ? acc + per_round * (3 + 2 * NB) : acc);
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
  q.acc = acc;
  q.fix = fix;
  q.sw = p.sw;
  q.status = p.status;
  int dev = 0, nsm = 0;
  RR_CUDA_TRY(cudaGetDevice(&dev));
  RR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
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
                              p.tm.igm_model, w.pix_stride, basis, GRAD ? dbasis : nullptr, bad,
                              p.status, st);
    if (rc) return rc;
    p.pair_target = all.pair_target + i0;
    p.chi2 = all.chi2 + i0;
    p.coeff = all.coeff + i0 * NB;
    p.penalty = all.penalty ? all.penalty + i0 : nullptr;
    if (GRAD) {
      p.dchi2_dz = all.dchi2_dz + i0;
      p.d2chi2_dz2 = all.d2chi2_dz2 + i0;
      p.dpen_dz = all.dpen_dz ? all.dpen_dz + i0 : nullptr;
      q.dflux = all.dchi2_dflux ? all.dchi2_dflux + i0 * p.npix_row : nullptr;
    }
    q.pair_target = p.pair_target;
    q.n = n;
    q.coeff = p.coeff;
    q.chi2 = p.chi2;
    q.dbasis = nullptr;
    rc = launch_sums<NB, false>(q, st);
    if (rc) return rc;
    pairs_solve_kernel<NB, GRAD><<<(unsigned)((n + 63) / 64), 64, 0, st>>>(p, my, bad, n, fix);
    RR_CHECK_LAUNCH();
    if constexpr (GRAD) {
      q.dbasis = dbasis;
      rc = launch_sums<NB, true>(q, st);
      if (rc) return rc;
      pairs_slope_kernel<NB><<<(unsigned)((n + 63) / 64), 64, 0, st>>>(p, my, acc, n, fix);
    } else {
      const int64_t rg = n < (int64_t)nsm * 8 ? n : (int64_t)nsm * 8;
      pairs_resid_kernel<NB><<<(unsigned)rg, kPairThreads, 0, st>>>(q);
    }
    RR_CHECK_LAUNCH();
  }
  return RR_OK;
}

// the call's rounds: nearly equal, within the builder's grid (the arrays of any
// number of pairs are aligned: basis rows are an even number of doubles)
template <bool GRAD>
static int run_pairs_ws(const PairsParams& p, const rr_pair_segment* segs, void* workspace,
                        size_t workspace_bytes, cudaStream_t st) {
  if (!workspace ||
      ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(p.rows)) & 15))
    return RR_EINVAL;
  const PairsWsLayout w = pairs_ws_layout(segs, p.nseg, p.tm.nbasis, GRAD);
  int64_t most = (int64_t)(workspace_bytes / (size_t)w.per_pair);
  if (most < 1) return RR_EINVAL;
  if (most > 65534 * build_z(false)) most = 65534 * build_z(false);
  const int64_t rounds = (p.npairs + most - 1) / most;
  const int64_t per_round = (p.npairs + rounds - 1) / rounds;
  int rc = basis_tables(st);
  if (rc) return rc;
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  switch (p.tm.nbasis) {
    case 1: return launch_pairs_ws<1, GRAD>(p, w, ws, per_round, st);
    case 2: return launch_pairs_ws<2, GRAD>(p, w, ws, per_round, st);
    case 3: return launch_pairs_ws<3, GRAD>(p, w, ws, per_round, st);
    case 4: return launch_pairs_ws<4, GRAD>(p, w, ws, per_round, st);
    case 5: return launch_pairs_ws<5, GRAD>(p, w, ws, per_round, st);
    case 6: return launch_pairs_ws<6, GRAD>(p, w, ws, per_round, st);
    case 7: return launch_pairs_ws<7, GRAD>(p, w, ws, per_round, st);
    case 8: return launch_pairs_ws<8, GRAD>(p, w, ws, per_round, st);
    case 9: return launch_pairs_ws<9, GRAD>(p, w, ws, per_round, st);
    case 10: return launch_pairs_ws<10, GRAD>(p, w, ws, per_round, st);
    default: return RR_EINVAL;
  }
}

}  // namespace rr

using namespace rr;

static bool pair_segments_ok(const rr_pair_segment* segs, int nseg) {
  if (!segs || nseg < 1 || nseg > kPairMaxSeg) return false;
  for (int s = 0; s < nseg; ++s)
    if (segs[s].npix < 1) return false;
  return true;
}

static size_t ws_bytes(const rr_pair_segment* segs, int nseg, int32_t nbasis, int64_t npairs,
                       bool grad) {
  if (!pair_segments_ok(segs, nseg) || nbasis < 1 || nbasis > RR_MAX_NBASIS || npairs < 0)
    return SIZE_MAX;
  size_t b = 0;
  if (__builtin_mul_overflow((size_t)pairs_ws_layout(segs, nseg, nbasis, grad).per_pair,
                             (size_t)npairs, &b))
    return SIZE_MAX;
  return b;
}

extern "C" size_t rr_zscan_pairs_ws_bytes(const rr_pair_segment* segs, int nseg, int32_t nbasis,
                                          int64_t npairs) {
  return ws_bytes(segs, nseg, nbasis, npairs, false);
}

extern "C" size_t rr_zscan_pairs_grad_ws_bytes(const rr_pair_segment* segs, int nseg,
                                               int32_t nbasis, int64_t npairs) {
  return ws_bytes(segs, nseg, nbasis, npairs, true);
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
  return run_pairs_ws<false>(p, segs, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int rr_zscan_pairs_grad_ws(const rr_pair_template* tmpl, const rr_pair_segment* segs,
                                      int nseg, const double* rows, const double* sw,
                                      const double* fwf, const double* wsum, int64_t npix_row,
                                      const int32_t* pair_target, const double* pair_z,
                                      int64_t npairs, double* chi2, double* coeff,
                                      double* penalty, double* dchi2_dz, double* d2chi2_dz2,
                                      double* dchi2_dflux, double* dpenalty_dz, void* workspace,
                                      size_t workspace_bytes, int* status, rr_stream_t stream) {
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
  return run_pairs_ws<true>(p, segs, workspace, workspace_bytes, (cudaStream_t)stream);
}
