// Small frames: one launch, a thread per path, as the megakernel, with the
// four-wide walks at 128 registers (170 where lights of every shape, textures
// or bump maps are compiled in), where they do not spill.  The staged renderer
// (path_stages.cuh) launches two kernels a bounce, each as long as the bounce's
// longest walk; where a frame's paths fit a wave or two of warps, the longest
// path alone is shorter.  The megakernel's code, so the film is its film to the
// bit.
//
// A warp's paths are an 8x4 tile of pixels, and frames that would leave the SMs
// short of warps put fewer paths into each, whose lanes then wait for fewer
// other lanes' walks.
#pragma once
#include "integrator.cuh"
#include "kernels.h"
#include "megakernel.cuh"

namespace nb {

template <int ISECT, bool EXT, bool DIFF>
__global__ void __launch_bounds__(kMegaBlock, kSmallBlocks(EXT)) small_frames(DevScene S, DevCamera C, MegaArgs a,
                                                                              uint32_t lanes) {
    extern __shared__ uint32_t smem[];
    const uint32_t npix = C.w * C.h;
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x, lane = thread & 31u;
    const uint32_t idx = (thread >> 5) * lanes + lane;
    RayStats rs{0u, 0u};
    uint32_t paths = 0;
    if (lane < lanes && idx < npix * a.nframes) {
        const uint32_t pix = stage_pixel(idx % npix, C.w, C.h), f = idx / npix, frame = a.frame0 + f;
        SmemStack st{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
        Rng rng{tea16(pix, frame)};
        float3 o, d, hitp = f3(0.0f);
        RayDiff rd{};
        if (DIFF)
            camera_ray_diff(C, pix % C.w, pix / C.w, rng, o, d, rd);
        else
            camera_ray<EXT>(C, pix % C.w, pix / C.w, rng, o, d);
        const bool want_hit = pix == C.center && f + 1u == a.nframes;
        bool hit_valid = false;
        const float3 L = path_radiance<ISECT, EXT, DIFF, true>(S, o, d, rng, st, a.status, rs,
                                                               want_hit ? &hitp : nullptr, &hit_valid, rd);
        paths = 1;
        if (S.film_mode != NOOR_FILM_KAHAN) {
            // one frame (the launch's condition)
            const float4 old = frame > 1u && !a.fresh ? a.film_sum[pix] : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            const float t = 1.0f / (float)frame;
            a.film_sum[pix] = make_float4(old.x + t * (L.x - old.x), old.y + t * (L.y - old.y),
                                          old.z + t * (L.z - old.z), old.w + t * (1.0f - old.w));
        } else {
            float3 sum = f3(0.0f), comp = f3(0.0f);
            if (a.chunks == 1u && !a.fresh) {
                sum = f3(a.film_sum[pix]);
                comp = f3(a.film_comp[pix]);
            }
            kahan_add(sum, comp, L);
            const bool film = a.chunks == 1u;
            (film ? a.film_sum : a.part_sum)[film ? pix : (size_t)f * npix + pix] =
                make_float4(sum.x, sum.y, sum.z, film ? 1.0f : 0.0f);
            (film ? a.film_comp : a.part_comp)[film ? pix : (size_t)f * npix + pix] =
                make_float4(comp.x, comp.y, comp.z, 0.0f);
        }
        if (want_hit) *a.lookat = make_float4(hitp.x, hitp.y, hitp.z, hit_valid ? 1.0f : 0.0f);
    }
    warp_count(a.counters + 0, rs.ext);
    warp_count(a.counters + 1, rs.shadow);
    warp_count(a.counters + 2, paths);
}

template <int ISECT>
cudaError_t launch_small_isect(const DevScene& S, const DevCamera& C, const MegaArgs& a, uint32_t lanes, cudaStream_t s) {
    const uint32_t warps = (C.w * C.h * a.nframes + lanes - 1u) / lanes;
    const uint32_t grid = (warps + kMegaBlock / 32 - 1) / (kMegaBlock / 32);
    const size_t sm = (size_t)S.stack_words * kMegaBlock * sizeof(uint32_t);
    auto go = [&](auto kern) {
        cudaError_t e = allow_stacks(kern, kMegaBlock);
        if (e != cudaSuccess) return e;
        kern<<<grid, kMegaBlock, sm, s>>>(S, C, a, lanes);
        return cudaGetLastError();
    };
    if (S.has_bump) return go(small_frames<ISECT, true, true>);
    return ext_kernels(S, C) ? go(small_frames<ISECT, true, false>) : go(small_frames<ISECT, false, false>);
}

}  // namespace nb
