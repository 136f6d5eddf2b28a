// The plain megakernel (one path per (pixel, frame),
// noor/cuda/path_tracer.cu:77-100) and its launch for one intersector; each
// intersector's kernels are compiled in a file of their own.  It walks the
// binary tree: inlined into the path loop at 72 registers the four-wide walk
// spills (1920x1080 sky frame 3.59 -> 3.78 ms, textured room 4.0 -> 5.1).
#pragma once
#include "integrator.cuh"
#include "kernels.h"

namespace nb {

// warp-aggregated add of per-lane counts into a 64-bit device counter
NB_D void warp_count(unsigned long long* ctr, uint32_t v) {
    const uint32_t mask = __activemask();
    const uint32_t s = __reduce_add_sync(mask, v);
    const int leader = __ffs(mask) - 1;
    if ((int)(threadIdx.x & 31) == leader && s) atomicAdd(ctr, (unsigned long long)s);
}

NB_D void kahan_add(float3& sum, float3& c, const float3& x) {
    const float3 y = x - c;
    const float3 t = sum + y;
    c = (t - sum) - y;
    sum = t;
}

// minimum resident blocks per SM the megakernel is compiled for: 7 caps its
// registers at 65536 / (128 * 7) = 73, i.e. 28 warps per SM instead of 12
// at its natural ~155 registers; the traversal is latency-bound, so the
// occupancy is worth the spilled values (measured faster on the sky-lit
// 2.6M-triangle scene than 5 or 6)
#ifndef NB_MEGA_MIN_BLOCKS
#define NB_MEGA_MIN_BLOCKS 7
#endif

template <int ISECT, int FILM, bool EXT, bool DIFF = false>
__global__ void __launch_bounds__(kMegaBlock, NB_MEGA_MIN_BLOCKS) megakernel(DevScene S, DevCamera C, MegaArgs a) {
    extern __shared__ uint32_t smem[];
    const uint32_t npix = C.w * C.h;
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t pix = idx % npix;
    const uint32_t chunk = idx / npix;
    RayStats rs{0u, 0u};
    uint32_t paths = 0;
    if (chunk < a.chunks) {
        const uint32_t per = (a.nframes + a.chunks - 1) / a.chunks;
        const uint32_t fb = chunk * per;
        const uint32_t fe = min(fb + per, a.nframes);
        SmemStack st{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
        const uint32_t x = pix % C.w, y = pix / C.w;
        float3 sum = f3(0.0f), comp = f3(0.0f);
        float4 mean = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        if (a.chunks == 1u && !a.fresh) {
            if (FILM == NOOR_FILM_KAHAN) {
                sum = f3(a.film_sum[pix]);
                comp = f3(a.film_comp[pix]);
            } else {
                mean = a.film_sum[pix];
            }
        }
        float3 hitp = f3(0.0f);
        bool hit_valid = false;
        const bool want_hit = (pix == C.center) && (chunk == a.chunks - 1u);
        for (uint32_t f = fb; f < fe; ++f) {
            const uint32_t frame = a.frame0 + f;
            Rng rng{tea16(pix, frame)};
            float3 o, d;
            RayDiff rd{};
            if (DIFF)
                camera_ray_diff(C, x, y, rng, o, d, rd);
            else
                camera_ray<EXT>(C, x, y, rng, o, d);
            hit_valid = false;
            const float3 L = path_radiance<ISECT, EXT, DIFF>(S, o, d, rng, st, a.status, rs,
                                                             want_hit ? &hitp : nullptr, &hit_valid, rd);
            ++paths;
            if (FILM == NOOR_FILM_KAHAN) {
                kahan_add(sum, comp, L);
            } else {
                // framebuffer.set: lerp(old, new, 1/frame) (framebuffer.cuh:72-76)
                const float4 old = frame > 1u ? mean : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
                const float t = 1.0f / (float)frame;
                mean = make_float4(old.x + t * (L.x - old.x), old.y + t * (L.y - old.y), old.z + t * (L.z - old.z),
                                   old.w + t * (1.0f - old.w));
            }
        }
        if (a.chunks == 1u) {
            if (FILM == NOOR_FILM_KAHAN) {
                a.film_sum[pix] = make_float4(sum.x, sum.y, sum.z, 1.0f);
                a.film_comp[pix] = make_float4(comp.x, comp.y, comp.z, 0.0f);
            } else {
                a.film_sum[pix] = mean;
            }
        } else {
            const size_t o = (size_t)chunk * npix + pix;
            a.part_sum[o] = make_float4(sum.x, sum.y, sum.z, 0.0f);
            a.part_comp[o] = make_float4(comp.x, comp.y, comp.z, 0.0f);
        }
        if (want_hit) *a.lookat = make_float4(hitp.x, hitp.y, hitp.z, hit_valid ? 1.0f : 0.0f);
    }
    warp_count(a.counters + 0, rs.ext);
    warp_count(a.counters + 1, rs.shadow);
    warp_count(a.counters + 2, paths);
}

// scenes without the extra lobes and lights, seen through a pinhole, run a
// specialisation without the other code (the kernel's registers are capped,
// so unused branches cost spills)
template <int ISECT>
cudaError_t launch_megakernel_isect(const DevScene& S, const DevCamera& C, const MegaArgs& a, cudaStream_t s) {
    const uint64_t threads = (uint64_t)C.w * C.h * a.chunks;
    const uint32_t grid = (uint32_t)((threads + kMegaBlock - 1) / kMegaBlock);
    const size_t sm = (size_t)S.stack_cap * kMegaBlock * sizeof(uint32_t);
    const bool ext = ext_kernels(S, C);
    auto go = [&](auto kern) {
        cudaError_t e = allow_stacks(kern, kMegaBlock);
        if (e != cudaSuccess) return e;
        kern<<<grid, kMegaBlock, sm, s>>>(S, C, a);
        return cudaGetLastError();
    };
    if (S.film_mode == NOOR_FILM_KAHAN) {
        if (S.has_bump) return go(megakernel<ISECT, NOOR_FILM_KAHAN, true, true>);
        if (ext) return go(megakernel<ISECT, NOOR_FILM_KAHAN, true, false>);
        return go(megakernel<ISECT, NOOR_FILM_KAHAN, false, false>);
    }
    if (S.has_bump) return go(megakernel<ISECT, NOOR_FILM_REF_LERP, true, true>);
    if (ext) return go(megakernel<ISECT, NOOR_FILM_REF_LERP, true, false>);
    return go(megakernel<ISECT, NOOR_FILM_REF_LERP, false, false>);
}

}  // namespace nb
