#include "small_frames.cuh"

namespace nb {

cudaError_t launch_small_frames_wt(const DevScene& S, const DevCamera& C, const MegaArgs& a, uint32_t lanes,
                                   cudaStream_t s) {
    return launch_small_isect<NOOR_ISECT_WATERTIGHT>(S, C, a, lanes, s);
}

}  // namespace nb
