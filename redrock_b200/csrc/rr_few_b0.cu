// Scan of a few targets: bounded solves, nbasis 1..7 (rr_few.cuh).
#include "rr_few.cuh"

namespace rr {

int few_bounded_lo(int nbasis, FewParams& p, const rr_scan_template* templates, const int* pick,
                   int npick, bool overlap, cudaStream_t stream) {
#define RR_FEW_CASE(N) \
  case N:              \
    return launch_few<N, true>(p, templates, pick, npick, overlap, stream);
  switch (nbasis) {
    RR_FEW_CASE(1) RR_FEW_CASE(2) RR_FEW_CASE(3) RR_FEW_CASE(4) RR_FEW_CASE(5) RR_FEW_CASE(6)
    RR_FEW_CASE(7)
    default: return RR_EINVAL;
  }
#undef RR_FEW_CASE
}

}  // namespace rr
