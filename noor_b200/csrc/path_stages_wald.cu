// The staged renderer's kernels with the reference's Wald triangle test
#include "path_stages_launch.cuh"

namespace nb {
cudaError_t launch_stages_wald(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                             cudaStream_t s) {
    return launch_stages<NOOR_ISECT_REF_WALD>(S, C, W, sm_count, launches, s);
}
}  // namespace nb
