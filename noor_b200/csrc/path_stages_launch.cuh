// Launches of the staged renderer's kernels for one intersector
#pragma once
#include <algorithm>

#include "path_stages.cuh"

namespace nb {

template <int ISECT, bool EXT, bool DIFF>
cudaError_t run_stages(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                       cudaStream_t s) {
    constexpr int trav = 64;
    const size_t sm = (size_t)S.stack_words * trav * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(st_trace<ISECT, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    const uint32_t all = (W.paths + 255) / 256;
    const uint32_t gt = std::min<uint32_t>((W.paths + trav - 1) / trav, (uint32_t)sm_count * 16);
    const dim3 gs(std::min<uint32_t>((W.paths + 127) / 128, (uint32_t)sm_count * 8), kStageKinds);
    st_begin<EXT, DIFF><<<all, 256, 0, s>>>(C, W);
    st_trace<ISECT, EXT><<<gt, trav, sm, s>>>(S, C, W, -1);
    for (uint32_t b = 0; b < S.bounces; ++b) {
        st_shade<ISECT, EXT, DIFF><<<gs, 128, 0, s>>>(S, W, b);
        st_trace<ISECT, EXT><<<dim3(gt, 2), trav, sm, s>>>(S, C, W, (int)b);
    }
    *launches += 3 + 2 * (uint64_t)S.bounces;
    st_finish<ISECT, EXT><<<all, 256, 0, s>>>(S, W);
    return cudaGetLastError();
}

template <int ISECT>
cudaError_t launch_stages(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                          cudaStream_t s) {
    const bool ext_cam = C.type != NOOR_CAMERA_PERSP || C.lens_radius > 0.0f;
    if (S.has_bump) return run_stages<ISECT, true, true>(S, C, W, sm_count, launches, s);
    if (S.ext_lobes || S.ext_lights || S.env_ref || S.has_tex || ext_cam)
        return run_stages<ISECT, true, false>(S, C, W, sm_count, launches, s);
    return run_stages<ISECT, false, false>(S, C, W, sm_count, launches, s);
}

}  // namespace nb
