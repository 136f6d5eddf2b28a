// Launches of the staged renderer's kernels for one intersector
#pragma once
#include <algorithm>

#include "path_stages.cuh"

namespace nb {

constexpr int kStageTrav = 64, kStageTraceBlocks = 14;  // st_trace: 7 blocks of 128 threads in registers

template <int ISECT, bool EXT, bool DIFF>
cudaError_t run_stages(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                       cudaStream_t s) {
    const size_t sm = (size_t)S.stack_words * kStageTrav * sizeof(uint32_t);
    cudaError_t e = allow_stacks(st_trace<ISECT, EXT>, kStageTrav);
    if (e != cudaSuccess) return e;
    const uint32_t all = (W.paths + 255) / 256;
    // Two paths a warp until there are paths enough, where a walk is all that a
    // ray does; 32 a warp where lights of every shape and alpha maps come into
    // it, whose code then runs on fewer SMs (one sample of a 128x96 frame, 2 /
    // 4 / 16 / 32 a warp: room 178 / 179 / 189 / 209 us, textured room 324 /
    // 324 / 261 / 270; 192x144: 202 to 216, and 373 / 377 / 360 / 294)
    constexpr uint32_t kPer = EXT ? 64 : 4;
    const uint32_t gt = std::min<uint32_t>((W.paths + kPer - 1) / kPer, (uint32_t)(sm_count * kStageTraceBlocks));
    const uint32_t gs = std::min<uint32_t>((W.paths + 127) / 128, (uint32_t)sm_count * (EXT ? 4 : 6));
    if ((e = launch_stage(st_begin<EXT, DIFF>, all, 256, 0, s, C, W)) ||
        (e = launch_stage(st_trace<ISECT, EXT>, gt, kStageTrav, sm, s, S, C, W, -1)))
        return e;
    *launches += 3;
    for (uint32_t b = 0; b < S.bounces; ++b) {
        if (b && b % kStageAsk == 0 && S.bounces - b >= kStageAsk) {
            uint32_t left = 0;
            if ((e = cudaMemcpyAsync(&left, W.count + b * kStWords + kStActive, 4, cudaMemcpyDeviceToHost, s)) ||
                (e = cudaStreamSynchronize(s)))
                return e;
            if (left == 0) break;
        }
        if ((e = launch_stage(st_shade<ISECT, EXT, DIFF>, gs, 128, 0, s, S, W, b)) ||
            (e = launch_stage(st_trace<ISECT, EXT>, gt, kStageTrav, sm, s, S, C, W, (int)b)))
            return e;
        *launches += 2;
    }
    return launch_stage(st_finish<ISECT, EXT>, all, 256, 0, s, S, W);
}

template <int ISECT>
cudaError_t launch_stages(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                          cudaStream_t s) {
    if (S.has_bump) return run_stages<ISECT, true, true>(S, C, W, sm_count, launches, s);
    if (ext_kernels(S, C))
        return run_stages<ISECT, true, false>(S, C, W, sm_count, launches, s);
    return run_stages<ISECT, false, false>(S, C, W, sm_count, launches, s);
}

}  // namespace nb
