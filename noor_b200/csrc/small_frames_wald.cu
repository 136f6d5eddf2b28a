#include "small_frames.cuh"

namespace nb {

cudaError_t launch_small_frames_wald(const DevScene& S, const DevCamera& C, const MegaArgs& a, uint32_t lanes,
                                   cudaStream_t s) {
    return launch_small_isect<NOOR_ISECT_REF_WALD>(S, C, a, lanes, s);
}

}  // namespace nb
