// Basis builder: trapezoidal rebinning of template bases onto camera pixel
// bins for every redshift, fused with the IGM (Lyman-series) transmission.
//
// Reference behaviour followed (redrock 0.22):
//   _trapz_rebin_1d     rebin.py:126-176   (per-bin walk over input samples)
//   _trapz_rebin_batch  rebin.py:178-209   (x * (1 + z) per redshift)
//   trapz_rebin         rebin.py:212-378   (range check, output layout)
//   Inoue14             igm.py:105-267     (LAF/DLA series + continuum)
//   CaluraKamble        igm.py:321-364
//   DistTemplate        templates.py:584-597 (rebin, then data *= T)
//
// Design: one thread per output bin computes every basis of that bin, the
// basis builder for several redshifts in turn.  The first input sample beyond
// the bin's lower edge is found by a guess and a short walk on the redshifted
// grid (the reference walks it sequentially; both land on the first j with
// x[j](1+z) > edge).  All arithmetic of the rebin
// uses explicitly rounded operations in the reference's order, so results
// are bit-identical to redrock's CPU path.  The IGM factor of the bin's
// centre wavelength is computed in the same thread and multiplied in.
#include "rr_build.cuh"
#include "rr_rebin_dev.cuh"

namespace rr {

__global__ void igm_kernel(int model, const double* __restrict__ z, int64_t nz,
                           const double* __restrict__ lobs, int64_t nwave, double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t iz = blockIdx.y;
  if (i >= nwave || iz >= nz) return;
  out[iz * nwave + i] = transmission(model, z[iz], lobs[i]);
}

// out[(iz * z_stride) + ibin * bin_stride + b]
__global__ void trapz_rebin_kernel(const double* __restrict__ x, int64_t nx,
                                   const double* __restrict__ y, int nb,
                                   const double* __restrict__ edges, int64_t nbin,
                                   const double* __restrict__ z, int64_t nz, double* __restrict__ out,
                                   int64_t z_stride, int64_t bin_stride, int* status) {
  const int64_t ibin = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t iz = blockIdx.y;
  if (ibin >= nbin || iz >= nz) return;
  const double zp1 = dadd(1.0, z[iz]);
  double res[kMaxRebinBasis];
  double* o = out + iz * z_stride + ibin * bin_stride;
  if (!rebin_bin(x, nx, y, nb, zp1, edges[ibin], edges[ibin + 1], res)) {
    set_status(status, RR_ERANGE);
    for (int b = 0; b < nb; ++b) o[b] = nan("");
    return;
  }
  for (int b = 0; b < nb; ++b) o[b] = res[b];
}

template <int NB, bool DZ>
__device__ __noinline__ bool rebin_bin_general(const double* __restrict__ x, int64_t nx,
                                               const double* __restrict__ y, double zp1,
                                               double e_lo, double e_hi, double (&res)[NB],
                                               double (&dres)[DZ ? NB : 1]) {
  double v[kMaxRebinBasis], dv[DZ ? kMaxRebinBasis : 1];
  if (!rebin_bin_strided<DZ>(x, nx, y, nx, NB, zp1, e_lo, e_hi, v, dv)) return false;
#pragma unroll
  for (int b = 0; b < NB; ++b) res[b] = v[b];
  if (DZ)
#pragma unroll
    for (int b = 0; b < NB; ++b) dres[b] = dv[b];
  return true;
}

// The same for up to ten bases in registers (rebin_bin_reg); a warp's rows
// leave through shared memory as one contiguous run.
template <int NB>
__global__ void __launch_bounds__(128) trapz_rebin_reg_kernel(
    const double* __restrict__ x, int64_t nx, const double* __restrict__ y,
    const double* __restrict__ edges, int64_t nbin, const double* __restrict__ z,
    double* __restrict__ out, int* status) {
  __shared__ double stage[128 * NB];
  const int64_t ibin = blockIdx.x * (int64_t)128 + threadIdx.x;
  const int64_t iz = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double res[NB], none[1];
  if (ibin < nbin) {
    const double zp1 = dadd(1.0, z[iz]);
    const double lo = edges[ibin], hi = edges[ibin + 1];
    bool exact = true;
    bool in = rebin_bin_reg<NB>(x, nx, y, nx, zp1, lo, hi, first_above(x, nx, zp1, lo), res, exact,
                                none);
    if (in && !exact) in = rebin_bin_general<NB, false>(x, nx, y, zp1, lo, hi, res, none);
    if (!in) {
      set_status(status, RR_ERANGE);
#pragma unroll
      for (int b = 0; b < NB; ++b) res[b] = nan("");
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) stage[threadIdx.x * NB + b] = res[b];
  }
  __syncwarp();
  const int64_t first = blockIdx.x * (int64_t)128 + warp * 32;
  const int n = (int)(nbin - first < 32 ? (nbin > first ? nbin - first : 0) : 32) * NB;
  double* o = out + (iz * nbin + first) * NB;
  for (int q = lane; q < n; q += 32) o[q] = stage[warp * 32 * NB + q];
}

// Fused builder for one grid: rebin + IGM into the padded basis layout.
// Threads cover the padded pixel range [pix_offset - 5, pix_offset +
// npix_pad + 5); pixels outside [pix_offset, pix_offset + npix) and basis
// columns >= nb are written as 0 so the scan's halo reads see zeros.
// This general form (any nb up to kMaxRebinBasis, any basis stride) serves
// what build_basis_kernel below has no instantiation for.
__global__ void build_basis_any_kernel(const double* __restrict__ x, int64_t nx,
                                       const double* __restrict__ y, int nb,
                                       const double* __restrict__ z, int64_t nz,
                                       const double* __restrict__ edges,
                                       const double* __restrict__ wave, int64_t npix,
                                       int64_t npix_pad, int64_t pix_offset, int igm_model,
                                       int apply_igm, double* __restrict__ basis,
                                       int64_t pix_stride, int basis_stride, int* status) {
  const int64_t span = npix_pad + 2 * kHalfBand;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // 0..span-1
  const int64_t iz = blockIdx.y;
  if (i >= span || iz >= nz) return;
  const int64_t ipix = i - kHalfBand;  // pixel index within the grid
  double* o = basis + (iz * pix_stride + pix_offset + ipix) * basis_stride;
  if (ipix < 0 || ipix >= npix) {
    for (int b = 0; b < basis_stride; ++b) o[b] = 0.0;
    return;
  }
  const double zz = z[iz];
  const double zp1 = dadd(1.0, zz);
  double res[kMaxRebinBasis];
  if (!rebin_bin(x, nx, y, nb, zp1, edges[ipix], edges[ipix + 1], res)) {
    set_status(status, RR_ERANGE);
    for (int b = 0; b < basis_stride; ++b) o[b] = nan("");
    return;
  }
  if (apply_igm) {
    const double t = transmission(igm_model, zz, wave[ipix]);
    for (int b = 0; b < nb; ++b) res[b] = dmul(res[b], t);
  }
  for (int b = 0; b < nb; ++b) o[b] = res[b];
  for (int b = nb; b < basis_stride; ++b) o[b] = 0.0;
}

static __device__ __noinline__ double transmission_plain(int model, double z, double lobs) {
  return transmission(model, z, lobs);
}

// d/dz of the Inoue14 factor t (the other models' is 0 between their steps)
static __device__ __noinline__ double transmission_slope(double t, double z, double lobs) {
  return -t * dtau_lc_dz_inoue14(z, lobs);
}

// The builder for basis rows of NB values (rounded up to even), all grids in
// one launch: a block takes 128 padded pixels and up to build_z redshifts, a
// thread one pixel for all of them, with the bases in registers.  What a pixel
// and what a redshift need of the IGM is then formed once (InoueWave, InoueZ)
// instead of once per (z, pixel) -- 16 redshifts to a block with Inoue14, 4
// without, where more would only leave the last wave of blocks emptier, and
// fewer than 16 on short redshift grids (build_per_block) --, the divisions
// share their reciprocals (rebin_bin_reg) and the rows leave through shared
// memory as whole 16-byte columns of a warp's 32 consecutive rows.
// Per (z, pixel, basis) about 35 FP64 operations at two samples to a bin (135
// with three full divisions).  Bound by its sample loads: L1 77 % busy, the
// FP64 pipe 46 % (QSO with Inoue14 45 and 47 %: latency).  GALAXY, 3311 x 7958 x 10: 3.60 -> 1.86 ms; QSO with
// Inoue14, 3794 x 7958 x 4: 2.14 -> 1.24 ms (build_basis_any_kernel, one
// thread per (z, pixel), before).
constexpr int kBuildThreads = 128;

struct BuildParams {
  const double* x;
  int64_t nx;
  const double* y;
  const double* z;
  int64_t nz;
  BuildGrid g[kBuildGrids];
  int first[kBuildGrids + 1];  // first block of each grid
  int ngrid;
  int igm_model;
  int kz;  // redshifts per block with Inoue14
  double* basis;
  double* dbasis;  // dT/dz in the same layout (DZ)
  int64_t pix_stride;
  int* bad;       // per redshift: 1 where a bin fell outside the template, or NULL
  int* status;    // RR_ERANGE there, or NULL
};

// Blocks per SM: small bases with Inoue14 are bound by the latency of its
// chains (QSO 1.53 ms at three, 1.34 at four, 1.24 at six), without it, and
// for large ones, fewer registers cost more (five STAR bases 8 % at six;
// GALAXY 1.92 / 1.85 / 2.83 ms).
constexpr int build_blocks(int nb, bool inoue, bool dz) {
  return dz ? 3 : (nb <= 5 && inoue ? 6 : 4);
}

// INOUE: the Inoue14 factor; else the other models, or none.  DZ: dT/dz too.
template <int NB, bool INOUE, bool DZ>
__global__ void __launch_bounds__(kBuildThreads, build_blocks(NB, INOUE, DZ)) build_basis_kernel(
    const __grid_constant__ BuildParams p) {
  constexpr int S = (NB + 1) & ~1;
  constexpr int kZ = build_z(INOUE);
  __shared__ __align__(16) double stage[kBuildThreads * S];
  __shared__ InoueZ zc[INOUE ? kZ : 1];
  __shared__ int s_igm[kZ];
  int ig = 0;
  while (ig + 1 < p.ngrid && (int)blockIdx.x >= p.first[ig + 1]) ++ig;
  const BuildGrid& gd = p.g[ig];
  const int64_t bx = blockIdx.x - p.first[ig];
  const int64_t span = gd.npix_pad + 2 * kHalfBand;
  const int64_t i = bx * kBuildThreads + threadIdx.x;
  const int per = INOUE ? p.kz : kZ;
  const int z0 = (int)blockIdx.y * per;
  const int nz = p.nz - z0 < per ? (int)(p.nz - z0) : per;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < nz) {
    // which redshifts of the block take the factor, and their powers of 1 + z
    const double zz = p.z[z0 + threadIdx.x];
    const bool want = gd.igm && p.igm_model != RR_IGM_NONE &&
                      !(ddiv(gd.wave_min, dadd(1.0, zz)) > kLyA);
    s_igm[threadIdx.x] = want;
    if (INOUE && want) zc[threadIdx.x] = inoue_z(zz);
  }
  __syncthreads();
  const int64_t ipix = i - kHalfBand;
  const bool real = ipix >= 0 && ipix < gd.npix;
  double e_lo = 0.0, e_hi = 0.0;
  InoueWave wv;
  wv.lobs = 0.0;
  if (real) {
    e_lo = gd.edges[ipix];
    e_hi = gd.edges[ipix + 1];
    if (gd.igm) wv.lobs = gd.wave[ipix];
  }
  const double x0 = p.x[0];
  const double per_x = (double)(p.nx - 1) / (p.x[p.nx - 1] - x0);
  // rows of this warp that exist
  const int64_t first = bx * kBuildThreads + warp * 32;
  const int nrow = (int)(span - first < 32 ? (span - first > 0 ? span - first : 0) : 32);
  double* row = stage + threadIdx.x * S;
  for (int k = 0; k < nz; ++k) {
    const int64_t iz = z0 + k;
    double res[NB], dres[DZ ? NB : 1];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      res[b] = 0.0;
      if (DZ) dres[b] = 0.0;
    }
    if (real) {
      const double zz = p.z[iz];
      const double zp1 = dadd(1.0, zz);
      const int64_t j =
          first_above_near(p.x, p.nx, zp1, e_lo, (e_lo * __drcp_rn(zp1) - x0) * per_x);
      bool exact = true;
      bool in = rebin_bin_reg<NB, DZ>(p.x, p.nx, p.y, p.nx, zp1, e_lo, e_hi, j, res, exact, dres);
      if (in && !exact)
        in = rebin_bin_general<NB, DZ>(p.x, p.nx, p.y, zp1, e_lo, e_hi, res, dres);
      if (!in) {
        set_status(p.status, RR_ERANGE);
        if (p.bad) p.bad[iz] = 1;
#pragma unroll
        for (int b = 0; b < NB; ++b) res[b] = nan("");
      } else if (s_igm[k]) {
        const double t = INOUE ? transmission_inoue14(zc[INOUE ? k : 0], wv)
                               : transmission_plain(p.igm_model, zz, wv.lobs);
        if (DZ) {
          const double dt = INOUE ? transmission_slope(t, zz, wv.lobs) : 0.0;
#pragma unroll
          for (int b = 0; b < NB; ++b) dres[b] = dres[b] * t + res[b] * dt;
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) res[b] = dmul(res[b], t);
      }
    }
#pragma unroll
    for (int d = 0; d < (DZ ? 2 : 1); ++d) {
#pragma unroll
      for (int b = 0; b < NB; ++b) row[b] = d ? dres[DZ ? b : 0] : res[b];
      if (NB & 1) row[S - 1] = 0.0;
      __syncwarp();
      const double2* src = reinterpret_cast<const double2*>(stage + warp * 32 * S);
      double2* dst = reinterpret_cast<double2*>(
          (d ? p.dbasis : p.basis) + (iz * p.pix_stride + gd.pix_offset - kHalfBand + first) * S);
#pragma unroll
      for (int c = 0; c < S / 2; ++c) {
        const int q = c * 32 + lane;
        if (q < nrow * (S / 2)) dst[q] = src[q];
      }
      __syncwarp();
    }
  }
}

// Redshifts per block: build_z where the grid then still holds two waves of
// blocks; fewer on shorter redshift grids with Inoue14, which would leave SMs
// idle behind the serial chain of a block.  QSO with Inoue14 (us, 16 to a block
// / this rule / one thread per (z, pixel)): 8 redshifts 73 / 46 / 62, 16 97 / 50
// / 60, 32 99 / 58 / 64, 64 103 / 77 / 83, 100 105 / 91 / 105, 300 163 / 161 /
// 216.  Without it 4 to a block are within 8 us of the best at any length.
static int build_per_block(const BuildParams& p, int nb, bool inoue, int nsm) {
  const int most = build_z(inoue);
  if (!inoue) return most;
  const int64_t two_waves = 2 * (int64_t)nsm * build_blocks(nb, true, p.dbasis != nullptr);
  const int64_t kz = p.nz * p.first[p.ngrid] / two_waves;
  return kz < 1 ? 1 : kz < most ? (int)kz : most;
}

template <int NB>
static int launch_build(BuildParams& p, cudaStream_t stream) {
  bool igm = false;
  for (int g = 0; g < p.ngrid; ++g) igm = igm || p.g[g].igm;
  const bool inoue = igm && p.igm_model == RR_IGM_INOUE14;
  int dev = 0, nsm = 0;
  RR_CUDA_TRY(cudaGetDevice(&dev));
  RR_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  p.kz = build_per_block(p, NB, inoue, nsm);
  dim3 grid((unsigned)p.first[p.ngrid], (unsigned)((p.nz + p.kz - 1) / p.kz));
  if (p.dbasis && inoue)
    build_basis_kernel<NB, true, true><<<grid, kBuildThreads, 0, stream>>>(p);
  else if (p.dbasis)
    build_basis_kernel<NB, false, true><<<grid, kBuildThreads, 0, stream>>>(p);
  else if (inoue)
    build_basis_kernel<NB, true, false><<<grid, kBuildThreads, 0, stream>>>(p);
  else
    build_basis_kernel<NB, false, false><<<grid, kBuildThreads, 0, stream>>>(p);
  RR_CHECK_LAUNCH();
  return RR_OK;
}

int build_basis_rows(const double* x, int64_t nx, const double* y, int nbasis, const double* z,
                     int64_t nz, const BuildGrid* grids, int ngrid, int igm_model,
                     int64_t pix_stride, double* basis, double* dbasis, int* bad, int* status,
                     cudaStream_t stream) {
  BuildParams p{};
  p.dbasis = dbasis;
  p.x = x;
  p.nx = nx;
  p.y = y;
  p.z = z;
  p.nz = nz;
  p.igm_model = igm_model;
  p.basis = basis;
  p.pix_stride = pix_stride;
  p.bad = bad;
  p.status = status;
  for (int g0 = 0; g0 < ngrid; g0 += kBuildGrids) {
    p.ngrid = ngrid - g0 < kBuildGrids ? ngrid - g0 : kBuildGrids;
    int64_t n = 0;
    for (int g = 0; g < p.ngrid; ++g) {
      p.g[g] = grids[g0 + g];
      p.first[g] = (int)n;
      n += (p.g[g].npix_pad + 2 * kHalfBand + kBuildThreads - 1) / kBuildThreads;
      if (n > INT32_MAX) return RR_EINVAL;
    }
    p.first[p.ngrid] = (int)n;
    int rc = RR_OK;
    switch (nbasis) {
      case 1: rc = launch_build<1>(p, stream); break;
      case 2: rc = launch_build<2>(p, stream); break;
      case 3: rc = launch_build<3>(p, stream); break;
      case 4: rc = launch_build<4>(p, stream); break;
      case 5: rc = launch_build<5>(p, stream); break;
      case 6: rc = launch_build<6>(p, stream); break;
      case 7: rc = launch_build<7>(p, stream); break;
      case 8: rc = launch_build<8>(p, stream); break;
      case 9: rc = launch_build<9>(p, stream); break;
      case 10: rc = launch_build<10>(p, stream); break;
      default: return RR_EINVAL;
    }
    if (rc) return rc;
  }
  return RR_OK;
}

int basis_tables(cudaStream_t stream) { return upload_igm_tables(stream); }

}  // namespace rr

using namespace rr;

extern "C" int rr_trapz_rebin(const double* x, int64_t nx, const double* y, int64_t nbasis,
                              const double* edges, int64_t nbin, const double* z, int64_t nz,
                              double xmin, double xmax, double edge_min, double edge_max,
                              double* out, int* status, rr_stream_t stream) {
  if (nx < 2 || nbasis < 1 || nbasis > kMaxRebinBasis || nbin < 1 || nz < 0) return RR_EINVAL;
  if (!x || !y || !edges || (nz > 0 && (!z || !out))) return RR_EINVAL;
  if (edge_min < xmin || edge_max > xmax) return RR_ERANGE;
  if (nz == 0) return RR_OK;
  if (nz > 65535) return RR_ENOTSUP;
  dim3 block(128);
  dim3 grid((unsigned)((nbin + block.x - 1) / block.x), (unsigned)nz);
  cudaStream_t st = (cudaStream_t)stream;
#define RR_REBIN_CASE(N)                                                                          \
  case N:                                                                                         \
    trapz_rebin_reg_kernel<N><<<grid, block, 0, st>>>(x, nx, y, edges, nbin, z, out, status);     \
    break;
  switch (nbasis) {
    RR_REBIN_CASE(1) RR_REBIN_CASE(2) RR_REBIN_CASE(3) RR_REBIN_CASE(4) RR_REBIN_CASE(5)
    RR_REBIN_CASE(6) RR_REBIN_CASE(7) RR_REBIN_CASE(8) RR_REBIN_CASE(9) RR_REBIN_CASE(10)
    default:
      trapz_rebin_kernel<<<grid, block, 0, st>>>(x, nx, y, (int)nbasis, edges, nbin, z, nz, out,
                                                 nbin * nbasis, nbasis, status);
  }
#undef RR_REBIN_CASE
  RR_CHECK_LAUNCH();
  return RR_OK;
}

extern "C" int rr_igm_transmission(int model, const double* z, int64_t nz, const double* lobs,
                                   int64_t nwave, double* out, rr_stream_t stream) {
  if (model < RR_IGM_NONE || model > RR_IGM_INOUE14) return RR_EINVAL;
  if (nz < 0 || nwave < 0) return RR_EINVAL;
  if (nz == 0 || nwave == 0) return RR_OK;
  if (!z || !lobs || !out) return RR_EINVAL;
  if (nz > 65535) return RR_ENOTSUP;
  int rc = upload_igm_tables((cudaStream_t)stream);
  if (rc) return rc;
  dim3 block(128);
  dim3 grid((unsigned)((nwave + block.x - 1) / block.x), (unsigned)nz);
  igm_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(model, z, nz, lobs, nwave, out);
  RR_CHECK_LAUNCH();
  return RR_OK;
}

extern "C" int rr_build_basis(const double* x, int64_t nx, const double* y, int64_t nbasis,
                              const double* z, int64_t nz, double xmin, double xmax,
                              const rr_grid_desc* grids, int ngrid, int igm_model,
                              int64_t pix_stride, int basis_stride, double* basis, int* status,
                              rr_stream_t stream) {
  if (nx < 2 || nbasis < 1 || nbasis > kMaxRebinBasis || nz < 0 || ngrid < 1 || !grids)
    return RR_EINVAL;
  if (basis_stride < nbasis || (basis_stride & 1)) return RR_EINVAL;
  if (igm_model < RR_IGM_NONE || igm_model > RR_IGM_INOUE14) return RR_EINVAL;
  if (nz > 65535) return RR_ENOTSUP;
  for (int g = 0; g < ngrid; ++g) {
    const rr_grid_desc& gd = grids[g];
    if (gd.npix < 1 || gd.npix_pad < gd.npix || (gd.npix_pad % RR_CHUNK) != 0) return RR_EINVAL;
    if (gd.pix_offset < kHalfBand || gd.pix_offset + gd.npix_pad + kHalfBand > pix_stride)
      return RR_EINVAL;
    if (gd.edge_min < xmin || gd.edge_max > xmax) return RR_ERANGE;
  }
  if (nz == 0) return RR_OK;
  int rc = upload_igm_tables((cudaStream_t)stream);
  if (rc) return rc;
  if (nbasis <= 10 && basis_stride == ((nbasis + 1) & ~1) &&
      (reinterpret_cast<uintptr_t>(basis) & 15) == 0) {
    for (int g0 = 0; g0 < ngrid; g0 += kBuildGrids) {
      BuildGrid bg[kBuildGrids];
      const int n = ngrid - g0 < kBuildGrids ? ngrid - g0 : kBuildGrids;
      for (int g = 0; g < n; ++g) {
        const rr_grid_desc& gd = grids[g0 + g];
        bg[g] = BuildGrid{gd.edges, gd.wave, gd.npix, gd.npix_pad, gd.pix_offset, NAN,
                          gd.apply_igm && igm_model != RR_IGM_NONE};
      }
      rc = build_basis_rows(x, nx, y, (int)nbasis, z, nz, bg, n, igm_model, pix_stride, basis,
                            nullptr, nullptr, status, (cudaStream_t)stream);
      if (rc) return rc;
    }
    return RR_OK;
  }
  for (int g = 0; g < ngrid; ++g) {
    const rr_grid_desc& gd = grids[g];
    const int64_t span = gd.npix_pad + 2 * kHalfBand;
    dim3 block(128);
    dim3 grid((unsigned)((span + block.x - 1) / block.x), (unsigned)nz);
    build_basis_any_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(
        x, nx, y, (int)nbasis, z, nz, gd.edges, gd.wave, gd.npix, gd.npix_pad, gd.pix_offset,
        igm_model, gd.apply_igm && igm_model != RR_IGM_NONE, basis, pix_stride, basis_stride,
        status);
    RR_CHECK_LAUNCH();
  }
  return RR_OK;
}
