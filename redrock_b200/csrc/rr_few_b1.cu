// Scan of a few targets: bounded solves, nbasis 8..10 (rr_few.cuh).
#include "rr_few.cuh"

namespace rr {

int few_bounded_hi(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
                   int npick, bool overlap, cudaStream_t stream) {
#define RR_FEW_CASE(N) \
  case N:              \
    return launch_few<N, true>(p, templates, pick, npick, overlap, stream);
  switch (nbasis) {
    RR_FEW_CASE(8) RR_FEW_CASE(9) RR_FEW_CASE(10)
    default: return RR_EINVAL;
  }
#undef RR_FEW_CASE
}

}  // namespace rr
