// Render and parity kernels: the film fold, ray-batch traversal and the
// device-routine evaluators used by the parity tests (the megakernel is in
// megakernel.cuh).
#include <type_traits>

#include "kernels.h"
#include "integrator.cuh"

namespace nb {

NB_D void kahan_add(float3& sum, float3& c, const float3& x) {
    const float3 y = x - c;
    const float3 t = sum + y;
    c = (t - sum) - y;
    sum = t;
}

// folds the per-chunk partial sums into the Kahan film in chunk order
__global__ void fold_partials(uint32_t npix, uint32_t chunks, uint32_t fresh, float4* film_sum, float4* film_comp,
                              const float4* part_sum, const float4* part_comp) {
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    float3 sum = f3(0.0f), comp = f3(0.0f);
    if (!fresh) {
        sum = f3(film_sum[pix]);
        comp = f3(film_comp[pix]);
    }
    for (uint32_t c = 0; c < chunks; ++c) {
        const size_t o = (size_t)c * npix + pix;
        kahan_add(sum, comp, f3(part_sum[o]));
        kahan_add(sum, comp, -1.0f * f3(part_comp[o]));
    }
    film_sum[pix] = make_float4(sum.x, sum.y, sum.z, 1.0f);
    film_comp[pix] = make_float4(comp.x, comp.y, comp.z, 0.0f);
}

// film -> mean rgba
__global__ void film_resolve(uint32_t npix, int mode, float inv_count, const float4* film_sum, float4* out) {
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    const float4 s = film_sum[pix];
    out[pix] = mode == NOOR_FILM_KAHAN ? make_float4(s.x * inv_count, s.y * inv_count, s.z * inv_count, 1.0f) : s;
}

// EXT false: the scene has no sphere, disk or delta lights and no textures.
// 7 blocks (72 registers) as the wavefront's walks: a million scattered rays
// on 2.6M triangles, closest and any hit, take 0.556 ms (8 blocks 0.585, 6
// 0.571, 5 0.579; 0.673 with the extra lights' code and no bound).
constexpr int kTraceMinBlocks = 7;
template <int ISECT, bool WIDE, bool EXT>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_trace_closest(DevScene S, const noor_ray* rays, noor_hit* hits,
                                                               size_t n, uint32_t* status) {
    extern __shared__ uint32_t smem[];
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    SmemStack st{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
    const noor_ray r = rays[i];
    float tmax = r.tmax;
    HitRec rec{0.0f, 0.0f, 0u, 0u, 0u};
    const HeldRay world{f3(r.org[0], r.org[1], r.org[2]), f3(r.dir[0], r.dir[1], r.dir[2])};
    const bool h = trace_primary<ISECT, EXT, WIDE>(S, world, tmax, rec, st, status);
    noor_hit o;
    o.t = tmax;
    o.tri_idx = rec.tri;
    o.ins_idx = rec.ins;
    o.material_type = rec.mtype;
    o.u = rec.u;
    o.v = rec.v;
    o.hit = h ? 1u : 0u;
    o.pad = 0u;
    hits[i] = o;
}

template <int ISECT, bool WIDE, bool EXT>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_trace_any(DevScene S, const noor_ray* rays, uint32_t* occ,
                                                           size_t n, uint32_t* status) {
    extern __shared__ uint32_t smem[];
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    SmemStack st{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
    const noor_ray r = rays[i];
    const HeldRay world{f3(r.org[0], r.org[1], r.org[2]), f3(r.dir[0], r.dir[1], r.dir[2])};
    occ[i] = trace_shadow<ISECT, EXT, WIDE>(S, world, r.tmax, st, status) ? 1u : 0u;
}

__global__ void k_camera_rays(DevCamera C, uint32_t frame, noor_ray* rays) {
    const uint32_t npix = C.w * C.h;
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    Rng rng{tea16(pix, frame)};
    float3 o, d;
    camera_ray(C, pix % C.w, pix / C.w, rng, o, d);
    noor_ray r;
    r.org[0] = o.x;
    r.org[1] = o.y;
    r.org[2] = o.z;
    r.tmax = kInf;
    r.dir[0] = d.x;
    r.dir[1] = d.y;
    r.dir[2] = d.z;
    r.pad = 0.0f;
    rays[pix] = r;
}

// in: {wo[3], wi[3], u[2], mat, 0..} (16 floats) in the local frame whose
// geometric and shading normals are +z; out: {f[3], pdf, wi[3], type}
__global__ void k_eval_bsdf(DevScene S, int kind, const float* in, float* out, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* p = in + 16 * i;
    const float3 wo = f3(p[0], p[1], p[2]);
    const float3 wi = f3(p[3], p[4], p[5]);
    const uint32_t mi = (uint32_t)p[8];
    const DevMaterial m = S.materials[mi];
    Frame F;
    F.n = f3(0.0f, 0.0f, 1.0f);
    F.ng = F.n;
    F.s = f3(1.0f, 0.0f, 0.0f);
    F.t = f3(0.0f, 1.0f, 0.0f);
    const uint32_t lobe = lobe_of(m.type);
    float* q = out + 8 * i;
    float3 f = f3(0.0f), wo_s = f3(0.0f);
    float pdf = 0.0f;
    uint32_t st = 0;
    if (kind == 0) {
        f = bsdf_eval(lobe, m, F, wo, wi, BSDF_ALL);
    } else if (kind == 1) {
        pdf = bsdf_pdf(lobe, m, F, wo, wi, BSDF_ALL);
    } else {
        // the BSDF's Sample_f with its two uniforms given (no RNG)
        float3 w = f3(0.0f);
        f = bsdf_sample_u(lobe, m, F, wo, BSDF_ALL, p[6], p[7], w, pdf, st);
        if (pdf != 0.0f) wo_s = w;
    }
    q[0] = f.x;
    q[1] = f.y;
    q[2] = f.z;
    q[3] = pdf;
    q[4] = wo_s.x;
    q[5] = wo_s.y;
    q[6] = wo_s.z;
    q[7] = (float)st;
}

// Stand-alone shading routines for parity tests; record layouts in
// include/noor_b200.h (noor_eval_routines).
__global__ void k_eval_routines(int kind, const float* in, float* out, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (kind <= 1) {
        const float* p = in + 12 * i;
        float* q = out + 12 * i;
        Micro m;
        m.ax = fmaxf(p[0] * p[0], 1e-3f);
        m.ay = fmaxf(p[1] * p[1], 1e-3f);
        m.dist = (uint32_t)kind;
        const float3 wo = f3(p[2], p[3], p[4]), wh = f3(p[5], p[6], p[7]);
        const float3 s = m.sample_wh(wo, p[8], p[9]);
        const float r[12] = {m.D(wh), m.G(wo, wh), m.pdf(wo, wh), s.x, s.y, s.z, 0.0f, m.ax, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int k = 0; k < 12; ++k) q[k] = r[k];
    } else if (kind == 2) {
        const float* p = in + 9 * i;
        float* q = out + 4 * i;
        q[0] = fresnel_dielectric(p[0], p[1], p[2]);
        const float3 c = fresnel_conductor(p[0], f3(p[3], p[4], p[5]), f3(p[6], p[7], p[8]));
        q[1] = c.x;
        q[2] = c.y;
        q[3] = c.z;
    } else {
        const float* p = in + 3 * i;
        float* q = out + 16 * i;
        const float2 d = concentric_disk(p[0], p[1]);
        const float3 c = cosine_hemisphere(p[0], p[1]);
        float st;
        const float3 sd = spherical_direction(p[0], p[1], st);
        const float3 h = uniform_hemisphere(p[0], p[1]);
        const float r[16] = {d.x, d.y, c.x, c.y, c.z, h.x, h.y, h.z, sd.x, sd.y, sd.z, st,
                             power_heuristic(p[0], p[1]), erf_as(p[2]), erfinv_giles(p[2]), 0.0f};
        for (int k = 0; k < 16; ++k) q[k] = r[k];
    }
}

__global__ void k_eval_sky(DevScene S, const float* dirs, float* rgb, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 c = env_eval<true>(S, f3(dirs[3 * i], dirs[3 * i + 1], dirs[3 * i + 2]));
    rgb[3 * i] = c.x;
    rgb[3 * i + 1] = c.y;
    rgb[3 * i + 2] = c.z;
}

// u -> {x, y, pdf_sample, pdf_eval}
__global__ void k_env_sample(DevScene S, const float* u, float* out, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float pdf;
    const float2 xy = S.env_ref ? rdist_sample(S, u[2 * i], u[2 * i + 1], pdf) : dist_sample(S.dist, u[2 * i], u[2 * i + 1], pdf);
    out[4 * i] = xy.x;
    out[4 * i + 1] = xy.y;
    out[4 * i + 2] = pdf;
    out[4 * i + 3] = S.env_ref ? rdist_pdf(S, xy.x, xy.y) : dist_pdf(S.dist, xy.x, xy.y);
}

// debug_skydome_kernel (noor/cuda/path_tracer.cu:102-122)
__global__ void k_debug_skydome(DevScene S, DevCamera C, uint32_t frame, float4* film, int mis) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= C.w || y >= C.h) return;
    const uint32_t id = y * C.w + x;
    const float u = x / (float)C.w, v = y / (float)C.h;
    float3 c;
    if (S.sky_type == NOOR_SKY_PHYSICAL) {
        float3 dir = f3(sinf(v * kPi) * cosf(u * k2Pi), cosf(v * kPi), sinf(v * kPi) * sinf(u * k2Pi));
        c = sinf(v * kPi) * hosek_query(S.hosek, normalize_fast(dir));
    } else {
        c = env_bilinear(S, u, v);
    }
    film[id] = make_float4(c.x, c.y, c.z, 1.0f);
    if (mis) {
        Rng rng{tea16(id, frame)};
        const float a = rng.next();
        const float b = rng.next();
        float pdf;
        const float2 s = dist_sample(S.dist, a, b, pdf);
        const uint32_t px = min((uint32_t)(s.x * C.w), C.w - 1), py = min((uint32_t)(s.y * C.h), C.h - 1);
        film[py * C.w + px] = make_float4(1.0f, 0.0f, 0.0f, 1.0f);
    }
}

// ------------------------------------------------------------ launchers
static cudaError_t launch_fold(const DevCamera& C, const MegaArgs& a, cudaStream_t s) {
    if (a.chunks <= 1u) return cudaSuccess;
    const uint32_t npix = C.w * C.h;
    fold_partials<<<(npix + 255) / 256, 256, 0, s>>>(npix, a.chunks, a.fresh, a.film_sum, a.film_comp, a.part_sum,
                                                      a.part_comp);
    return cudaGetLastError();
}

cudaError_t launch_megakernel(const DevScene& S, const DevCamera& C, const MegaArgs& a, cudaStream_t s) {
    const cudaError_t e =
        S.isect == NOOR_ISECT_WATERTIGHT ? launch_megakernel_wt(S, C, a, s) : launch_megakernel_wald(S, C, a, s);
    return e == cudaSuccess ? launch_fold(C, a, s) : e;
}

// The line between small frames (a thread per path) and the staged renderer.
// A staged bounce costs its longest walk and two launches whatever the frame,
// so the line rises with the bounces that a path can make and with the depth of
// the tree; beyond it the stages' fuller warps win.  In waves of resident
// threads, megakernel / stages / small frames in us:
//   1.5   36-triangle room, 384x288: 2 bounces 140 / 134 / 108, 8: 362 / 323 / 307
//         (448x336: 158 / 138 / 125 and 423 / 324 / 391); 2 bounces under the
//         sky, 384x288: 280 / 227 / 212 and 333 / 242 / 242 (448x336: 383 / 250 / 320)
//   4     8 bounces under the sky, 641x359: 164 k triangles 450 / 488 / 365 and
//         608 / 497 / 492, 2.6 M triangles 774 / 718 / 540 (800x450: 651 / 497 / 545,
//         851 / 816 / 664)
//   6-12  limits of 12 to 32 and more bounces, where a few paths that stay inside
//         glass cost the stages a walk and two launches each time: 800x450 under
//         five skies, limit 12, 609 / 670 / 387 to 901 / 564 / 730; 960x540, limit 128,
//         4593 / 5225 / 2701 and 4970 / 5447 / 3154 to 1291 / 683 / 1016
//   3     the room with a limit of 32, 384x288: 419 / 562 / 346 (512x512: 796 / 753 / 829)
//   1     with the code of all lights, textures and bump maps, 5 bounces in the
//         textured room: 192x144 329 / 291 / 271, 320x240 514 / 371 / 403
//   4.5   the same with limits of 16 and more, of 32: 384x288 788 / 1179 / 648, 641x359 984 / 1310 / 948
bool small_frames_fit(const DevScene& S, const DevCamera& C, const MegaArgs& a, int sm_count) {
    const bool ext = ext_kernels(S, C), shallow = S.num_tris < 16384u;
    const uint64_t wave = (uint64_t)sm_count * kSmallBlocks(ext) * kMegaBlock;
    const uint32_t b = S.bounces;
    const uint64_t half_waves = ext       ? (b < 8u ? 2 : b < 12u ? 3 : b < 16u ? 4 : 9)
                                : shallow ? (b < 12u ? 3 : b < 24u ? 4 : 6)
                                          : (b < 4u ? 3 : b < 6u ? 4 : b < 12u ? 8 : b < 16u ? 12 : b < 32u ? 16 : 24);
    return 2 * (uint64_t)C.w * C.h * a.nframes <= wave * half_waves;
}

cudaError_t launch_small_frames(const DevScene& S, const DevCamera& C, const MegaArgs& a, int sm_count, cudaStream_t s) {
    // trees without a four-wide form: the megakernel's walks
    if (!S.frames4) return launch_megakernel(S, C, a, s);
    // Paths a warp, a power of two: 32, or fewer where that leaves warps to
    // spare.  Walks fill the resident warps (one frame under the sky of 97x61,
    // 32 / 8 / 4 paths a warp: 147 / 115 / 102 us); the larger code of the
    // other lights and textures is bound by its instruction fetch from some
    // five warps per SM on (the textured room, 97x61: 130 / 107 / 128; 160x120,
    // 32 / 16: 161 / 183).
    const bool ext = ext_kernels(S, C);
    const uint64_t warps = (uint64_t)sm_count * (ext ? 5 : kSmallBlocks(ext) * (kMegaBlock / 32));
    const uint64_t paths = (uint64_t)C.w * C.h * a.nframes;
    uint32_t lanes = 32;
    while (lanes > 1u && paths <= warps * (lanes / 2)) lanes /= 2;
    const cudaError_t e = S.isect == NOOR_ISECT_WATERTIGHT ? launch_small_frames_wt(S, C, a, lanes, s)
                                                           : launch_small_frames_wald(S, C, a, lanes, s);
    return e == cudaSuccess ? launch_fold(C, a, s) : e;
}

cudaError_t launch_resolve(uint32_t npix, int mode, float inv_count, const float4* film_sum, float4* out,
                           cudaStream_t s) {
    film_resolve<<<(npix + 255) / 256, 256, 0, s>>>(npix, mode, inv_count, film_sum, out);
    return cudaGetLastError();
}

// one launch of a ray-batch kernel: the four-wide or the binary traversal,
// per intersector, with or without the extra lights' code
template <template <int, bool, bool> class K, class T>
static cudaError_t launch_trace(const DevScene& S, bool wide, const noor_ray* rays, T* out, size_t n,
                                uint32_t* status, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    // room for the four-wide tree's stacks as well as the binary one's
    const size_t sm = (size_t)S.stack_words * kTraceBlock * sizeof(uint32_t);
    const uint32_t grid = (uint32_t)((n + kTraceBlock - 1) / kTraceBlock);
    auto go = [&](auto kern) {
        cudaError_t e = allow_stacks(kern, kTraceBlock);
        if (e != cudaSuccess) return e;
        kern<<<grid, kTraceBlock, sm, s>>>(S, rays, out, n, status);
        return cudaGetLastError();
    };
    const bool ext = S.ext_lights || S.has_tex;
    auto pick = [&](auto isect) {
        constexpr int I = decltype(isect)::value;
        if (wide) return ext ? go(K<I, true, true>::fn) : go(K<I, true, false>::fn);
        return ext ? go(K<I, false, true>::fn) : go(K<I, false, false>::fn);
    };
    if (S.isect == NOOR_ISECT_WATERTIGHT) return pick(std::integral_constant<int, NOOR_ISECT_WATERTIGHT>());
    return pick(std::integral_constant<int, NOOR_ISECT_REF_WALD>());
}
template <int I, bool W, bool X>
struct ClosestK {
    static constexpr auto fn = k_trace_closest<I, W, X>;
};
template <int I, bool W, bool X>
struct AnyK {
    static constexpr auto fn = k_trace_any<I, W, X>;
};

cudaError_t launch_trace_closest(const DevScene& S, const noor_ray* rays, noor_hit* hits, size_t n, uint32_t* status,
                                 cudaStream_t s) {
    return launch_trace<ClosestK>(S, S.closest4 != 0u, rays, hits, n, status, s);
}

cudaError_t launch_trace_any(const DevScene& S, const noor_ray* rays, uint32_t* occ, size_t n, uint32_t* status,
                             cudaStream_t s) {
    return launch_trace<AnyK>(S, S.nodes4 != nullptr, rays, occ, n, status, s);
}

cudaError_t launch_camera_rays(const DevCamera& C, uint32_t frame, noor_ray* rays, cudaStream_t s) {
    const uint32_t npix = C.w * C.h;
    k_camera_rays<<<(npix + 255) / 256, 256, 0, s>>>(C, frame, rays);
    return cudaGetLastError();
}

cudaError_t launch_eval_bsdf(const DevScene& S, int kind, const float* in, float* out, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_eval_bsdf<<<(uint32_t)((n + 255) / 256), 256, 0, s>>>(S, kind, in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_eval_routines(int kind, const float* in, float* out, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_eval_routines<<<(uint32_t)((n + 255) / 256), 256, 0, s>>>(kind, in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_eval_sky(const DevScene& S, const float* dirs, float* rgb, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_eval_sky<<<(uint32_t)((n + 255) / 256), 256, 0, s>>>(S, dirs, rgb, n);
    return cudaGetLastError();
}

cudaError_t launch_env_sample(const DevScene& S, const float* u, float* out, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_env_sample<<<(uint32_t)((n + 255) / 256), 256, 0, s>>>(S, u, out, n);
    return cudaGetLastError();
}

cudaError_t launch_debug_skydome(const DevScene& S, const DevCamera& C, uint32_t frame, float4* film, int mis,
                                 cudaStream_t s) {
    dim3 b(16, 16), g((C.w + 15) / 16, (C.h + 15) / 16);
    k_debug_skydome<<<g, b, 0, s>>>(S, C, frame, film, mis);
    return cudaGetLastError();
}

}  // namespace nb
