// The staged renderer's kernels with the watertight triangle test
#include "path_stages_launch.cuh"

namespace nb {
cudaError_t launch_stages_wt(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                             cudaStream_t s) {
    return launch_stages<NOOR_ISECT_WATERTIGHT>(S, C, W, sm_count, launches, s);
}
}  // namespace nb
