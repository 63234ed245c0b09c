// The basis builder of rr_basis.cu, as the pair scan calls it.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace rr {

constexpr int kBuildGrids = 16;  // grids per launch

// redshifts per block of the builder, at most
__host__ __device__ constexpr int build_z(bool inoue) { return inoue ? 16 : 4; }

struct BuildGrid {
  const double* edges;
  const double* wave;
  int64_t npix, npix_pad, pix_offset;
  double wave_min;  // redshifts that leave it redward of Lyman-alpha get no
                    // IGM factor (it is exactly 1 there); NaN: no such rule
  int igm;          // 0: no factor on this grid
};

// Basis rows of nbasis (<= 10) values rounded up to even, 16-byte aligned, of
// nz redshifts on the given grids; the tables of basis_tables are uploaded.
// dbasis (or NULL) gets dT/dz in the same layout; bad[iz] = 1 and status RR_ERANGE where a bin falls outside the template.
int build_basis_rows(const double* x, int64_t nx, const double* y, int nbasis, const double* z,
                     int64_t nz, const BuildGrid* grids, int ngrid, int igm_model,
                     int64_t pix_stride, double* basis, double* dbasis, int* bad, int* status,
                     cudaStream_t stream);
int basis_tables(cudaStream_t stream);

}  // namespace rr
