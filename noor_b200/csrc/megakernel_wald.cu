// The megakernel with the reference's Wald triangle test
#include "megakernel.cuh"

namespace nb {
cudaError_t launch_megakernel_wald(const DevScene& S, const DevCamera& C, const MegaArgs& a, cudaStream_t s) {
    return launch_megakernel_isect<NOOR_ISECT_REF_WALD>(S, C, a, s);
}
}  // namespace nb
