// The megakernel with the watertight triangle test
#include "megakernel.cuh"

namespace nb {
cudaError_t launch_megakernel_wt(const DevScene& S, const DevCamera& C, const MegaArgs& a, cudaStream_t s) {
    return launch_megakernel_isect<NOOR_ISECT_WATERTIGHT>(S, C, a, s);
}
}  // namespace nb
