// Staged rendering of cuda_path_tracer / noor_render_frames: the megakernel's
// path loop cut into one launch per stage and bounce over every path of a
// batch of frames, so that traversal runs without the shading code's
// registers and shading runs over queues of one material kind.
//
//   begin    camera rays
//   per bounce:
//     extend  closest hit for the bounce's paths; surface hits are queued by
//             material kind
//     shade   the direct light of the last bounce folded into the path's
//             radiance, light (and MIS) samples whose shadow rays are queued,
//             scatter, Russian roulette, the next ray
//     shadow  any hit; blocked contributions are cancelled (in one launch with
//             the next bounce's extend)
//   finish   what is pending and the sky or emitter a path ended on
//   fold     each pixel's samples into the film, in frame order and with the
//            megakernel's split into chunks
//
// Every path draws the megakernel's random numbers and evaluates the
// megakernel's expressions in its order and with its rounding, so the film is
// the megakernel's to the bit.  The megakernel is bound by divergence (8-10 of
// 32 lanes: a warp runs until its longest path ends) and by instruction fetch;
// the stages run 13 and more lanes of small kernels.  Measured against the
// megakernel: 256x256 room 0.305 -> 0.248 ms, 1920x1080 of a 2.6M-triangle
// sky scene 3.68 -> 2.45, sixteen 960x540 frames of an environment-lit field
// 14.7 -> 4.06, four 641x359 frames of the textured room 3.98 -> 0.88.  Few
// paths are bound by latency, bounce after bounce: the stages are launched
// ahead of each other's end, and a bounce costs its longest walk, which falls on
// another path each time.  small_frames.cuh renders those frames.
#pragma once
#include "integrator.cuh"
#include "kernels.h"

namespace nb {

constexpr int kStageKinds = 3;  // shade_kind: Lambert, conductor, the rest

// Every path may have ended long before the bounce limit, and a bounce without
// paths takes 4 to 19 us (1920x1080 under the sky with a limit of 1024: 5.0 ms,
// of which 4.4 for nothing).  So every kStageAsk bounces, where as many are to
// come, the host asks what is left, which costs the launches' lead of some 20 us
// (512x512 room, 9 bounces: 472 us, 491 with the asking).
constexpr uint32_t kStageAsk = 8;

// counters of one bounce
enum : int {
    kStActive = kStageKinds,        // paths the bounce extends
    kStShadow = kStageKinds + 1,    // shadow rays queued
    kStTake = kStageKinds + 2,      // active paths taken by extend's warps
    kStTakeShadow = kStageKinds + 3,
    kStWords = 8
};

// how a path ended, beside the material types (hit2.y): nothing to add, or an
// escape to a sky it counts
constexpr uint32_t kStDone = 0x80000000u, kStSky = 0x40000000u;

struct StageDev {
    float4* o;          // origin
    float4* d;          // direction, w = 1 after a specular bounce
    float4* beta;       // throughput, w = 1 while contributions are pending
    float4* L;          // radiance, w = RNG state bits
    float4* pend;       // 2 per path: direct-light contribution, w = 1 while it counts
    float4* pbeta;      // the throughput it is weighted by
    float4* hit;        // t, u, v, triangle bits
    uint2* hit2;        // instance, material type or kSt*
    float4* diff;       // 4 per path where the scene has bump maps: the ray's differentials
    uint32_t* queue[2]; // paths of this bounce and of the next (bounce 0: all)
    uint32_t* qshade;   // kStageKinds * cap
    uint32_t* qshadow;  // 2 * cap: path << 1 | which
    float4* sh_o;       // origin, tmax
    float4* sh_d;
    uint32_t* count;    // kStWords per bounce, then one more
    float4* first;      // per frame of the batch: the centre pixel's first hit (w = 1)
    uint32_t* status;
    unsigned long long* counters;   // [ext rays, shadow rays, paths]
    uint32_t cap;       // queue stride
    uint32_t paths;     // paths of the batch
    uint32_t frames;    // frames of the batch
    uint32_t frame0;    // number of its first frame
    uint32_t zero;      // words from count to the end of first
    uint32_t keep;      // paths between the pend and pbeta entries of one bounce and the next (0: reused)
};

struct StageFold {
    uint32_t first;     // index of the batch's first frame in the call
    uint32_t total;     // frames of the call
    uint32_t chunks;
    uint32_t frame0;    // number of the call's first frame
    uint32_t fresh;
    uint32_t bounces;
    int film_mode;
    float4* film_sum;
    float4* film_comp;
    float4* part_sum;   // the running chunk's sum and compensation (chunks > 1)
    float4* part_comp;
    float4* lookat;
};

// warp-aggregated push: lanes of one warp may push onto different queues
NB_D uint32_t stage_push(uint32_t* counter) {
    const uint32_t active = __activemask();
    const uint32_t peers = __match_any_sync(active, reinterpret_cast<unsigned long long>(counter));
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(peers));
    base = __shfl_sync(active, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

NB_D void stage_store_diff(const StageDev& W, uint32_t i, const RayDiff& r) {
    W.diff[4 * i] = make_float4(r.odx.x, r.odx.y, r.odx.z, r.on ? 1.0f : 0.0f);
    W.diff[4 * i + 1] = make_float4(r.ody.x, r.ody.y, r.ody.z, 0.0f);
    W.diff[4 * i + 2] = make_float4(r.ddx.x, r.ddx.y, r.ddx.z, 0.0f);
    W.diff[4 * i + 3] = make_float4(r.ddy.x, r.ddy.y, r.ddy.z, 0.0f);
}
NB_D RayDiff stage_load_diff(const StageDev& W, uint32_t i) {
    const float4 a = W.diff[4 * i], b = W.diff[4 * i + 1], c = W.diff[4 * i + 2], e = W.diff[4 * i + 3];
    RayDiff r;
    r.on = a.w != 0.0f;
    r.odx = f3(a);
    r.ody = f3(b);
    r.ddx = f3(c);
    r.ddy = f3(e);
    return r;
}

// The stages are launched so that a kernel's blocks come to the SMs while the
// last blocks of the one before still run (programmatic stream serialization),
// and wait here until it has finished and its writes can be read.
NB_D void stage_follow() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

// kernel<<<g, b, sm, s>>>(args...), its blocks launched ahead of the end of
// the kernel before (stage_follow)
template <class... P, class... A>
cudaError_t launch_stage(void (*kernel)(P...), dim3 g, uint32_t b, size_t sm, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = g;
    c.blockDim = dim3(b);
    c.dynamicSmemBytes = sm;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// path i: pixel slot i / frames, frame i % frames (all samples of a pixel side by side)
template <bool EXT, bool DIFF>
__global__ void __launch_bounds__(256) st_begin(DevCamera C, StageDev W) {
    stage_follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // the batch's counters and first hits, which the stages after this one use
    for (uint32_t z = i; z < W.zero; z += gridDim.x * blockDim.x) W.count[z] = 0u;
    if (i >= W.paths) return;
    const uint32_t pix = stage_pixel(i / W.frames, C.w, C.h);
    Rng rng{tea16(pix, W.frame0 + i % W.frames)};
    float3 o, d;
    if (DIFF) {
        RayDiff rd{};
        camera_ray_diff(C, pix % C.w, pix / C.w, rng, o, d, rd);
        stage_store_diff(W, i, rd);
    } else {
        camera_ray<EXT>(C, pix % C.w, pix / C.w, rng, o, d);
    }
    W.o[i] = make_float4(o.x, o.y, o.z, 0.0f);
    W.d[i] = make_float4(d.x, d.y, d.z, 0.0f);
    W.beta[i] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    W.L[i] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(rng.s));
    W.hit2[i] = make_uint2(0u, kStDone);
}

// The next rays of a list of n for this warp.  The first rays of each of the
// launch's warps are its own by number, so that a short list takes no atomics
// and an empty one costs a warp one read; the rest are taken as warps get free.
NB_D uint32_t stage_take(uint32_t* taken, uint32_t warps, uint32_t take, uint32_t n, uint32_t lane) {
    if (warps * take >= n) return n;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(taken, take);
    return warps * take + __shfl_sync(0xFFFFFFFFu, base, 0);
}

template <int ISECT, bool EXT>
NB_D void stage_extend(const DevScene& S, const DevCamera& C, const StageDev& W, uint32_t bounce, const SmemStack& stk) {
    uint32_t* cnt = W.count + bounce * kStWords;
    const uint32_t n = bounce ? cnt[kStActive] : W.paths;
    const uint32_t* queue = W.queue[bounce & 1u];
    const uint32_t lane = threadIdx.x & 31, take = rays_per_warp(n);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    for (uint32_t base = warp * take; base < n; base = stage_take(cnt + kStTake, warps, take, n, lane)) {
        if (lane >= take || base + lane >= n) continue;
        const uint32_t i = bounce ? queue[base + lane] : base + lane;
        float tmax = kInf;
        HitRec rec{0.0f, 0.0f, 0u, 0u, 0u};
        const StoredRay ray{W.o + i, W.d + i};
        const bool binary = S.frames4 == 0u;
        if (!trace_closest4<ISECT, EXT>(S, ray, tmax, rec, stk, binary ? S.stack_cap : S.stack_cap4, binary, W.status)) {
            const bool sky = S.sky_on && (bounce == 0 || W.d[i].w != 0.0f);
            W.hit2[i] = make_uint2(0u, sky ? kStSky : kStDone);
            continue;
        }
        W.hit[i] = make_float4(tmax, rec.u, rec.v, __uint_as_float(rec.tri));
        uint32_t kind = rec.mtype;
        if (rec.mtype & kEmitterMat)
            // an emitter met by a bounce that does not count it adds nothing
            kind = bounce == 0 || W.d[i].w != 0.0f ? rec.mtype : kStDone;
        else
            W.qshade[shade_kind(lobe_of(rec.mtype)) * W.cap + stage_push(cnt + shade_kind(lobe_of(rec.mtype)))] = i;
        W.hit2[i] = make_uint2(rec.ins, kind);
        if (bounce == 0 && stage_pixel(i / W.frames, C.w, C.h) == C.center) {
            const float4 o = W.o[i], d = W.d[i];
            W.first[i % W.frames] = make_float4(fmaf(tmax, d.x, o.x), fmaf(tmax, d.y, o.y), fmaf(tmax, d.z, o.z), 1.0f);
        }
    }
}

// queues shadow ray `which` of path i; returns its place
NB_D uint32_t stage_shadow(const StageDev& W, uint32_t* cnt, uint32_t i, uint32_t which, const ShadowRay& sr) {
    const uint32_t k = stage_push(cnt + kStShadow);
    W.qshadow[k] = (i << 1) | which;
    W.sh_o[k] = make_float4(sr.o.x, sr.o.y, sr.o.z, sr.tmax);
    W.sh_d[k] = make_float4(sr.d.x, sr.d.y, sr.d.z, 0.0f);
    return k;
}

// the last bounce's direct light, as the megakernel adds it: L += beta * (c0 + c1)
NB_D void stage_pending(const StageDev& W, uint32_t i, float3& L) {
    const float4 p0 = W.pend[2 * i], p1 = W.pend[2 * i + 1], b = W.pbeta[i];
    float3 Ld = p0.w != 0.0f ? f3(p0) : f3(0.0f);
    if (p1.w != 0.0f) Ld += f3(p1);
    L += f3(b) * Ld;
}

// The queues of the material kinds one after the other, each filled up to
// whole warps, dealt to one wave of blocks: every warp shades one kind, a short
// queue shades beside a long one, and a bounce with nothing to shade costs one
// read a warp (three rows of 8 blocks per SM, a row per kind: 5.8 us for the
// empty bounces of a 768x512 frame, against 4.2 for st_trace's one wave).
// Bound by latency and by instruction fetch at these sizes: 4, 6 or 8 blocks
// per SM (16 to 32 warps) measure the same (1.10, 1.07, 1.09 ms for four
// 641x359 frames of the textured room); 6 leaves 80 registers.
template <int ISECT, bool EXT, bool DIFF>
__global__ void __launch_bounds__(128, EXT ? 4 : 6) st_shade(DevScene S, StageDev W, uint32_t bounce) {
    stage_follow();
    uint32_t* cnt = W.count + bounce * kStWords;
    const uint32_t n0 = cnt[0], n1 = cnt[1], n2 = cnt[2];
    const uint32_t b1 = (n0 + 31u) & ~31u, b2 = b1 + ((n1 + 31u) & ~31u);
    uint32_t* next = W.queue[(bounce & 1u) ^ 1u];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < b2 + n2; j += gridDim.x * blockDim.x) {
        const uint32_t kind_q = j < b1 ? 0u : j < b2 ? 1u : 2u;
        const uint32_t k = j - (kind_q == 0u ? 0u : kind_q == 1u ? b1 : b2);
        if (k >= (kind_q == 0u ? n0 : kind_q == 1u ? n1 : n2)) continue;
        const uint32_t i = W.qshade[kind_q * W.cap + k];
        const float4 ow = W.o[i], dw = W.d[i], bw = W.beta[i], Lw = W.L[i], hw = W.hit[i];
        const uint2 h2 = W.hit2[i];
        float3 L = f3(Lw), beta = f3(bw);
        if (bw.w != 0.0f) stage_pending(W, i, L);
        const float3 o = f3(ow), d = f3(dw);
        HitRec rec{hw.y, hw.z, __float_as_uint(hw.w), h2.x, h2.y};
        Isect I;
        TangentOut to;
        const bool tex = EXT && S.has_tex;
        make_isect<ISECT, EXT, true>(S, o, d, hw.x, rec, I, tex ? &to : nullptr);
        DevMaterial m = S.materials[I.mat];
        RayDiff rd{};
        HitDiff hd;
        if (DIFF) {
            rd = stage_load_diff(W, i);
            if (rd.on) {
                hd = hit_differential(I, to, rd);
                if (I.mtype & NOOR_BUMP) bump(S, I.mat, I.uv, hd, I.F);
            }
        }
        if (tex && m.tex_mask) apply_textures(S, I.mat, I.uv, m);
        Rng rng{__float_as_uint(Lw.w)};
        int li = 0;
        bool picked;
        ShadowRay sr;
        const float3 c0 = light_sample_contrib<EXT>(S, m, I, rng, S.mis != 0, li, picked, sr);
        const bool has0 = !is_black(c0);
        if (has0) stage_shadow(W, cnt, i, 0, sr);
        float3 c1 = f3(0.0f);
        bool has1 = false;
        if (S.mis && picked) {
            c1 = bsdf_mis_contrib<EXT>(S, m, I, rng, li, sr);
            has1 = !is_black(c1);
            if (has1) stage_shadow(W, cnt, i, 1, sr);
        }
        if (has0 || has1) {
            W.pend[2 * i] = make_float4(c0.x, c0.y, c0.z, has0 ? 1.0f : 0.0f);
            W.pend[2 * i + 1] = make_float4(c1.x, c1.y, c1.z, has1 ? 1.0f : 0.0f);
            W.pbeta[i] = make_float4(beta.x, beta.y, beta.z, 0.0f);
        } else {
            L += beta * 0.0f;  // as the megakernel: a throughput that is not finite ends the sample's radiance
        }
        rng.next();
        rng.next();
        float3 wi;
        float pdf;
        uint32_t stype;
        const float3 f = bsdf_sample<EXT>(I.lobe, m, I.F, I.wo, BSDF_ALL, rng, wi, pdf, stype);
        bool alive = pdf != 0.0f;
        if (alive) {
            beta *= (is_catcher<EXT>(I) ? f * catcher_sky<EXT>(S, I) : f) * absdot(wi, I.F.n) / pdf;
            if (!(I.mtype & kTransparentMat) && dot(wi, I.F.ng) < 0.0f) {
                alive = false;
            } else if (bounce >= S.rr) {
                const float q = fmaxf(0.05f, 1.0f - maxcomp(beta));
                if (rng.next() < q)
                    alive = false;
                else
                    beta /= 1.0f - q;
            }
        }
        if (alive) {
            const float3 no = spawn_origin(I, wi, S.bias);
            if (DIFF) {
                RayDiff nd{};
                if (rd.on && (I.mtype & kGlossyMat))
                    nd = spawn_diff(I, hd, rd, no, wi, (I.mtype & kDielectricMat) ? m.coat_ior : 1.0f);
                stage_store_diff(W, i, nd);
            }
            W.o[i] = make_float4(no.x, no.y, no.z, 0.0f);
            W.d[i] = make_float4(wi.x, wi.y, wi.z, (I.mtype & kSpecularMat) ? 1.0f : 0.0f);
            if (bounce + 1u < S.bounces) next[stage_push(cnt + kStWords + kStActive)] = i;
        }
        W.beta[i] = make_float4(beta.x, beta.y, beta.z, has0 || has1 ? 1.0f : 0.0f);
        W.L[i] = make_float4(L.x, L.y, L.z, __uint_as_float(rng.s));
        W.hit2[i].y = kStDone;
    }
}

template <int ISECT, bool EXT>
NB_D void stage_occlude(const DevScene& S, const StageDev& W, uint32_t bounce, const SmemStack& stk) {
    uint32_t* cnt = W.count + bounce * kStWords;
    const uint32_t n = cnt[kStShadow];
    const uint32_t lane = threadIdx.x & 31, take = rays_per_warp(n);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t warp = warps - 1u - (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    for (uint32_t base = warp * take; base < n; base = stage_take(cnt + kStTakeShadow, warps, take, n, lane)) {
        const uint32_t q = base + lane;
        if (lane >= take || q >= n) continue;
        const StoredRay ray{W.sh_o + q, W.sh_d + q};
        const bool binary = S.frames4 == 0u;
        if (trace_any4<ISECT, EXT>(S, ray, W.sh_o[q].w, stk, binary ? S.stack_cap : S.stack_cap4, binary, W.status))
            W.pend[2u * (size_t)W.keep * bounce + W.qshadow[q]].w = 0.0f;
    }
}

// The rays of a shade step: the next bounce's extension and the shadow rays,
// which only the next shade step waits for.  Every warp serves both lists, the
// extension first, and the lists are dealt out from the two ends of the grid,
// so that short lists meet on no warp.  One wave of blocks (kStageTraceBlocks
// per SM): a second one, or a row of blocks per list, only waits to find its
// list empty in the last bounces.
// bounce: the shade step's; extend only before the first (bounce -1) and
// shadow only after the last.
template <int ISECT, bool EXT>
__global__ void __launch_bounds__(128, 7) st_trace(DevScene S, DevCamera C, StageDev W, int bounce) {
    extern __shared__ uint32_t smem[];
    stage_follow();
    const SmemStack stk{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
    if (bounce + 1 < (int)S.bounces) stage_extend<ISECT, EXT>(S, C, W, (uint32_t)(bounce + 1), stk);
    if (bounce >= 0) stage_occlude<ISECT, EXT>(S, W, (uint32_t)bounce, stk);
}

// what a path's radiance still lacks; the clamped radiance into L
template <int ISECT, bool EXT>
__global__ void __launch_bounds__(256) st_finish(DevScene S, StageDev W) {
    stage_follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.paths) return;
    const float4 Lw = W.L[i], bw = W.beta[i];
    const uint2 h2 = W.hit2[i];
    float3 L = f3(Lw);
    const float3 beta = f3(bw);
    if (bw.w != 0.0f) stage_pending(W, i, L);
    if (h2.y == kStSky) {
        L += beta * env_eval<EXT>(S, f3(W.d[i]) * rsqrtf(stage_length2(f3(W.d[i]))));
    } else if (!(h2.y & kStDone)) {
        if (h2.y & NOOR_MESHLIGHT) {
            L += beta * area_le<EXT>(S.area_lights[h2.x], f3(W.d[i]));
        } else if (h2.y & kEmitterMat) {
            const float4 hw = W.hit[i];
            const uint32_t tri = __float_as_uint(hw.w);
            const uint32_t mi = ISECT == NOOR_ISECT_WATERTIGHT ? __ldg(&S.wtri[tri].attr).w : __ldg(&S.wald[tri].attr).w;
            DevMaterial em = S.materials[mi];
            if (EXT && S.has_tex && em.tex_mask) apply_textures(S, mi, f2(hw.y, hw.z), em);
            L += beta * (em.emitter_scale * em.emittance);
        }
    }
    L = clamp3(L, 0.0f, 100.0f);
    W.L[i] = make_float4(L.x, L.y, L.z, 0.0f);
}

}  // namespace nb
