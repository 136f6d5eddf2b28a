// The adjoint's replay cut into stages (adjoint.cu has the method and the form
// with a thread per path).
#include <algorithm>

#include "host_common.h"
// the replay's rounding of directions in the shading frame
#define NB_ADJOINT_ROUNDING
#include "adjoint.cuh"
#include "path_stages.cuh"

namespace nb {

// ------------------------------------------------------------- staged replay
// The replay cut into the stages of path_stages.cuh over the paths of a chunk
// of samples (camera rays, extension beside the last shadow rays, shading by
// material kind), with the expressions of `replay` and its rounding: the
// forward image is equal to the bit.  The backward pass records at every
// vertex what the gradient needs (RECORD), so that it walks no ray a second
// time; adj_backprop then goes through each path's vertices with its radiance
// known.  The thread-per-path kernels hold 128 and 165 registers and run a
// warp until its longest path ends, at 0.4 Grays/s; a 512x512, 16-sample,
// four-bounce step of forward and backward took 362 ms with them, 24.6 with
// the stages.
struct AdjStage {
    StageDev W;
    // records, vertex v of path i at v * W.keep + i
    float4* term_a;     // 2 per vertex: X s (f without its tint), dlog f / droughness
    float4* term_e;     // 2 per vertex: f s (light count), direction x
    float2* term_d;     // 2 per vertex: direction y, z
    float4* scatter;    // (f without its tint) / f, dlog f / droughness
    uint32_t* vertex;   // material and kAdj* bits
    uint32_t* count;    // vertices of path i
};
enum : uint32_t { kAdjMat = 0xFFFFu, kAdjEnv = 1u << 16 /* << term */, kAdjScatter = 1u << 18, kAdjRough = 1u << 19,
                  kAdjTint = 1u << 20 };

constexpr uint32_t kAdjNoRay = 0xFFFFFFFFu;

// direct_terms with the occlusion tests left to the shadow queue: term k's ray
// is queued as ray k of the path.  The two functions are alike to the
// statement, because the compiler's choice of fused multiply-adds follows the
// code around an expression, and a path must take the same turns in both.
template <int ISECT>
NB_D int queued_terms(const DevScene& S, const AdjParams& P, const StageDev& W, uint32_t* cnt, uint32_t i,
                      const DevMaterial& m0, const DevMaterial& me, const Isect& I, Rng& rng, Term* T, float3* dir) {
    int nt = 0;
    if (I.mtype & kSpecularMat) return 0;
    const int nl = S.sky_on ? S.num_lights : S.num_lights - 1;
    if (nl == 0) return 0;
    const int li = (int)((float)nl * rng.next());
    {
        float3 wi, to;
        float lpdf;
        const float3 Li0 = sample_li(S, I, rng, nl, li, wi, to, lpdf);
        if (lpdf != 0.0f && !is_black(Li0)) {
            const float3 f0 = bsdf_eval<false>(I.lobe, m0, I.F, I.wo, wi, kNonSpecular);
            if (!is_black(f0)) {
                const ShadowRay sr{spawn_origin(I, wi, S.bias), wi, 0.0f};
                const float tmax = length3(sr.o - to);
                if (stage_shadow(W, cnt, i, 0, ShadowRay{sr.o, sr.d, tmax}) != kAdjNoRay) {
                    dir[nt] = wi;
                    Term& t = T[nt++];
                    t.f = lobe_value(I.lobe, me, I.F, I.wo, wi);
                    float w = 1.0f;
                    if (S.mis) w = power_heuristic(lpdf, bsdf_pdf<false>(I.lobe, m0, I.F, I.wo, wi, kNonSpecular));
                    t.s = absdot(wi, I.F.n) * w / lpdf;
                    t.env = li >= S.num_area_lights && S.sky_type == NOOR_SKY_HDR;
                    t.xscale = (float)nl;
                    if (t.env) {
                        t.bl = env_weights(P, wi);
                        t.X = env_radiance(P, t.bl) * (float)nl;
                    } else {
                        t.X = Li0;
                    }
                }
            }
        }
    }
    if (!S.mis) return nt;
    rng.next();
    rng.next();
    float3 wi;
    float spdf;
    uint32_t stype;
    const float3 f0 = bsdf_sample<false>(I.lobe, m0, I.F, I.wo, kNonSpecular, rng, wi, spdf, stype);
    if (is_black(f0) || spdf == 0.0f) return nt;
    float w = 1.0f;
    if (!(stype & BSDF_SPECULAR)) {
        const float lp = light_pdf(S, I, li, wi);
        if (lp == 0.0f) return nt;
        w = power_heuristic(spdf, lp);
    }
    const float3 so = spawn_origin(I, wi, S.bias);
    float tm = 2.0f * S.world_radius;
    bool lh;
    float3 Le;
    const bool env = li >= S.num_area_lights;
    if (!env) {
        const DevAreaLight& A = S.area_lights[li];
        lh = quad_hit(A, so, wi, tm);
        Le = (A.two_sided || dot(wi, A.n) < 0.0f) ? A.ke : f3(0.0f);
    } else {
        lh = S.sky_on != 0;
        Le = S.sky_on ? env_eval<false>(S, wi) : f3(0.0f);
    }
    if (!lh || is_black(Le)) return nt;
    const float3 to = so + tm * wi;
    float3 vwi;
    visibility(I.p, to, vwi);
    const float3 so2 = spawn_origin(I, vwi, S.bias);
    if (stage_shadow(W, cnt, i, (uint32_t)nt, ShadowRay{so2, vwi, length3(so2 - to)}) == kAdjNoRay) return nt;
    dir[nt] = wi;
    Term& t = T[nt++];
    t.f = lobe_value(I.lobe, me, I.F, I.wo, wi);
    t.s = absdot(wi, I.F.n) * w / spdf;
    t.env = env && S.sky_type == NOOR_SKY_HDR;
    t.xscale = 1.0f;
    if (t.env) {
        t.bl = env_weights(P, wi);
        t.X = env_radiance(P, t.bl);
    } else {
        t.X = Le;
    }
    return nt;
}

NB_D void record_term(const AdjStage& A, size_t r, int k, const Term& t, const float3& wi) {
    const float3 xf = t.X * t.s * t.f.f_untinted, fe = t.f.f * (t.s * t.xscale);
    A.term_a[2 * r + k] = make_float4(xf.x, xf.y, xf.z, t.f.dlogf_dr);
    A.term_e[2 * r + k] = make_float4(fe.x, fe.y, fe.z, wi.x);
    A.term_d[2 * r + k] = make_float2(wi.y, wi.z);
}

__global__ void __launch_bounds__(256) adj_begin(DevCamera C, AdjStage A) {
    const StageDev& W = A.W;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.paths) return;
    const uint32_t pix = stage_pixel(i / W.frames, C.w, C.h);
    Rng rng{tea16(pix, W.frame0 + i % W.frames)};
    float3 o, d;
    camera_ray<false>(C, pix % C.w, pix / C.w, rng, o, d);
    W.o[i] = make_float4(o.x, o.y, o.z, 0.0f);
    W.d[i] = make_float4(d.x, d.y, d.z, 0.0f);
    W.beta[i] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    W.L[i] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(rng.s));
    W.hit2[i] = make_uint2(0u, kStDone);
    if (A.count) A.count[i] = 0u;
}

template <int ISECT>
__global__ void __launch_bounds__(128, 7) adj_trace(DevScene S, DevCamera C, StageDev W, int bounce) {
    extern __shared__ uint32_t smem[];
    const SmemStack stk{smem + threadIdx.x, (int)blockDim.x, S.stack_cap};
    if (blockIdx.y == 0) {
        if (bounce + 1 < (int)S.bounces) stage_extend<ISECT, false>(S, C, W, (uint32_t)(bounce + 1), stk);
    } else {
        stage_occlude<ISECT, false>(S, W, (uint32_t)bounce, stk);
    }
}

// the direct light of a vertex: the sum of its unoccluded terms (X f) s, each
// added as replay adds it (pend: X f, and s or zero)
NB_D float3 vertex_light(const StageDev& W, size_t r) {
    const float4 p0 = W.pend[2 * r], p1 = W.pend[2 * r + 1];
    float3 Ld = f3(0.0f);
    if (p0.w != 0.0f) Ld = f3(__fmul_rn(p0.x, p0.w), __fmul_rn(p0.y, p0.w), __fmul_rn(p0.z, p0.w));
    if (p1.w != 0.0f)
        Ld = f3(__fmaf_rn(p1.x, p1.w, Ld.x), __fmaf_rn(p1.y, p1.w, Ld.y), __fmaf_rn(p1.z, p1.w, Ld.z));
    return Ld;
}
NB_D void add_light(const StageDev& W, size_t r, float3& L) {
    const float3 b = f3(W.pbeta[r]), Ld = vertex_light(W, r);
    L = f3(__fmaf_rn(b.x, Ld.x, L.x), __fmaf_rn(b.y, Ld.y, L.y), __fmaf_rn(b.z, Ld.z, L.z));
}

template <int ISECT, bool RECORD>
__global__ void __launch_bounds__(128, 4) adj_shade(DevScene S, AdjParams P, AdjStage A, uint32_t bounce) {
    const StageDev& W = A.W;
    uint32_t* cnt = W.count + bounce * kStWords;
    const uint32_t kind_q = blockIdx.y, n = cnt[kind_q];
    uint32_t* next = W.queue[(bounce & 1u) ^ 1u];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t i = W.qshade[kind_q * W.cap + k];
        const size_t r = (size_t)W.keep * bounce + i;
        const float4 ow = W.o[i], dw = W.d[i], bw = W.beta[i], Lw = W.L[i], hw = W.hit[i];
        const uint2 h2 = W.hit2[i];
        float3 L = f3(Lw), beta = f3(bw);
        if (bw.w != 0.0f) add_light(W, r - W.keep, L);
        const float3 o = f3(ow), d = f3(dw);
        HitRec rec{hw.y, hw.z, __float_as_uint(hw.w), h2.x, h2.y};
        Isect I;
        make_isect<ISECT, false, true>(S, o, d, hw.x, rec, I);
        const DevMaterial m0 = S.materials[I.mat];
        const DevMaterial me = eval_material(m0, P, I.mat);
        Rng rng{__float_as_uint(Lw.w)};
        Term T[2];
        float3 dir[2];
        const int nt = queued_terms<ISECT>(S, P, W, cnt, i, m0, me, I, rng, T, dir);
        uint32_t word = I.mat;
        for (int k = 0; k < nt; ++k) {
            // (a scale of zero goes into the product: zero marks an occluded term)
            const bool zero = T[k].s == 0.0f;
            float3 v = T[k].X * T[k].f.f;
            if (zero) v = v * T[k].s;
            W.pend[2 * r + k] = make_float4(v.x, v.y, v.z, zero ? 1.0f : T[k].s);
            if (RECORD) {
                record_term(A, r, k, T[k], dir[k]);
                if (T[k].env) word |= kAdjEnv << k;
            }
        }
        const bool pend = nt > 0;
        if (!pend) L += beta * 0.0f;  // as the replay, where the throughput is not finite
        if (pend || RECORD) {
            for (int k = nt; k < 2; ++k) W.pend[2 * r + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            W.pbeta[r] = make_float4(beta.x, beta.y, beta.z, 0.0f);
        }
        rng.next();
        rng.next();
        float3 wi;
        float pdf;
        uint32_t stype;
        const float3 f0 = bsdf_sample<false>(I.lobe, m0, I.F, I.wo, BSDF_ALL, rng, wi, pdf, stype);
        const bool tint = I.lobe == kLobeLambert || I.lobe == kLobeConductor;
        if (tint) word |= kAdjTint;
        if (I.lobe == kLobeConductor) word |= kAdjRough;
        bool alive = false;
        do {
            if (pdf == 0.0f) break;
            float3 fe;
            FDeriv fd{f3(0.0f), f3(0.0f), 0.0f};
            if (stype & BSDF_SPECULAR) {
                fe = f0;
            } else {
                fd = lobe_value(I.lobe, me, I.F, I.wo, wi);
                fe = fd.f;
            }
            if (RECORD && !(stype & BSDF_SPECULAR) && tint) {
                word |= kAdjScatter;
                A.scatter[r] = make_float4(fe.x != 0.0f ? fd.f_untinted.x / fe.x : 0.0f,
                                           fe.y != 0.0f ? fd.f_untinted.y / fe.y : 0.0f,
                                           fe.z != 0.0f ? fd.f_untinted.z / fe.z : 0.0f, fd.dlogf_dr);
            }
            beta *= fe * absdot(wi, I.F.n) / pdf;
            if (!(I.mtype & kTransparentMat) && dot(wi, I.F.ng) < 0.0f) break;
            const float3 no = spawn_origin(I, wi, S.bias);
            W.o[i] = make_float4(no.x, no.y, no.z, 0.0f);
            W.d[i] = make_float4(wi.x, wi.y, wi.z, (I.mtype & kSpecularMat) ? 1.0f : 0.0f);
            alive = true;
        } while (false);
        if (alive && bounce + 1u < S.bounces) next[stage_push(cnt + kStWords + kStActive)] = i;
        W.beta[i] = make_float4(beta.x, beta.y, beta.z, pend ? 1.0f : 0.0f);
        W.L[i] = make_float4(L.x, L.y, L.z, __uint_as_float(rng.s));
        W.hit2[i].y = kStDone;
        if (RECORD) {
            A.vertex[r] = word;
            A.count[i] = bounce + 1u;
        }
    }
}

// what a path's radiance still lacks; sample-major into Lbuf for the forward
template <int ISECT>
__global__ void __launch_bounds__(256) adj_finish(DevScene S, DevCamera C, AdjParams P, AdjStage A, float4* Lbuf) {
    const StageDev& W = A.W;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.paths) return;
    const float4 Lw = W.L[i], bw = W.beta[i];
    const uint2 h2 = W.hit2[i];
    float3 L = f3(Lw);
    const float3 beta = f3(bw);
    if (bw.w != 0.0f) {
        const size_t last = W.keep ? (size_t)W.keep * (A.count[i] - 1u) : 0;
        add_light(W, last + i, L);
    }
    if (h2.y == kStSky) {
        const float3 d = f3(W.d[i]);
        const float3 dir = d * rsqrtf(stage_length2(d));
        float3 Le;
        if (S.sky_type == NOOR_SKY_HDR) {
            const Bilerp bl = env_weights(P, dir);
            Le = env_radiance(P, bl);
        } else {
            Le = env_eval<false>(S, dir);
        }
        L += beta * Le;
    } else if (!(h2.y & kStDone)) {
        if (h2.y & NOOR_MESHLIGHT) {
            const DevAreaLight& a = S.area_lights[h2.x];
            L += beta * ((a.two_sided || dot(f3(W.d[i]), a.n) < 0.0f) ? a.ke : f3(0.0f));
        } else if (h2.y & kEmitterMat) {
            const uint32_t tri = __float_as_uint(W.hit[i].w);
            const uint32_t mi = ISECT == NOOR_ISECT_WATERTIGHT ? __ldg(&S.wtri[tri].attr).w : __ldg(&S.wald[tri].attr).w;
            const DevMaterial& em = S.materials[mi];
            L += beta * (em.emitter_scale * em.emittance);
        }
    }
    if (Lbuf)
        Lbuf[(size_t)(i % W.frames) * (C.w * C.h) + stage_pixel(i / W.frames, C.w, C.h)] = make_float4(L.x, L.y, L.z, 0.0f);
    else
        W.L[i] = make_float4(L.x, L.y, L.z, 0.0f);
}

NB_D void add_texels(const AdjParams& P, const float3& dir, const float3& g) {
    const Bilerp bl = env_weights(P, dir);
    for (int k = 0; k < 4; ++k) {
        if (bl.w[k] == 0.0f) continue;
        float* e = P.g_env + 3 * bl.idx[k];
        atomicAdd(e + 0, g.x * bl.w[k]);
        atomicAdd(e + 1, g.y * bl.w[k]);
        atomicAdd(e + 2, g.z * bl.w[k]);
    }
}

// dLoss/dL of every path through the final clamp and on to the parameters,
// vertex by vertex (term_grad and the scattering step of replay<1>).  A warp
// adds the material gradients of its lanes per material before one lane adds
// them to the block's; resident blocks loop over the paths.
__global__ void __launch_bounds__(kAdjBlock) adj_backprop(DevScene S, DevCamera C, AdjParams P, AdjStage A) {
    __shared__ float sm[4 * kAdjMaxMats];   // albedo (3), roughness
    for (int i = threadIdx.x; i < 4 * kAdjMaxMats; i += blockDim.x) sm[i] = 0.0f;
    __syncthreads();
    const StageDev& W = A.W;
    const float inv_spp = 1.0f / (float)P.spp;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; b < W.paths; b += gridDim.x * blockDim.x) {
        const uint32_t i = b + lane;
        float3 dl = f3(0.0f), Lrem = f3(0.0f);
        uint32_t nv = 0;
        if (i < W.paths) {
            const uint32_t pix = stage_pixel(i / W.frames, C.w, C.h);
            const float3 gi = f3(P.grad_img[3 * pix], P.grad_img[3 * pix + 1], P.grad_img[3 * pix + 2]) * inv_spp;
            Lrem = f3(W.L[i]);
            dl = f3(Lrem.x > 0.0f && Lrem.x < 100.0f ? gi.x : 0.0f, Lrem.y > 0.0f && Lrem.y < 100.0f ? gi.y : 0.0f,
                    Lrem.z > 0.0f && Lrem.z < 100.0f ? gi.z : 0.0f);
            if (!is_black(dl)) {
                nv = A.count[i];
                if (W.hit2[i].y == kStSky && S.sky_type == NOOR_SKY_HDR) {
                    const float3 d = f3(W.d[i]);
                    add_texels(P, d * rsqrtf(stage_length2(d)), dl * f3(W.beta[i]));
                }
            }
        }
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, nv);
        for (uint32_t v = 0; v < most; ++v) {
            float3 ga = f3(0.0f);
            float gr = 0.0f;
            uint32_t mat = 0xFFFFFFFFu;
            if (v < nv) {
                const size_t r = (size_t)W.keep * v + i;
                const uint32_t word = A.vertex[r];
                const float3 g = dl * f3(W.pbeta[r]);
                for (uint32_t t = 0; t < 2; ++t) {
                    const float4 p = W.pend[2 * r + t];
                    if (p.w == 0.0f) continue;
                    const float4 ta = A.term_a[2 * r + t];
                    if (word & kAdjTint) {
                        ga += g * f3(ta);
                        if ((word & kAdjRough) && ta.w != 0.0f) {
                            const float3 q = g * f3(p) * p.w;
                            gr += (q.x + q.y + q.z) * ta.w;
                        }
                    }
                    if (word & (kAdjEnv << t)) {
                        const float4 te = A.term_e[2 * r + t];
                        const float2 td = A.term_d[2 * r + t];
                        add_texels(P, f3(te.w, td.x, td.y), g * f3(te));
                    }
                }
                Lrem = Lrem - f3(W.pbeta[r]) * vertex_light(W, r);
                if (word & kAdjScatter) {
                    const float4 sc = A.scatter[r];
                    const float3 h = dl * Lrem;
                    ga += h * f3(sc);
                    if ((word & kAdjRough) && sc.w != 0.0f) gr += (h.x + h.y + h.z) * sc.w;
                }
                if (ga.x != 0.0f || ga.y != 0.0f || ga.z != 0.0f || gr != 0.0f) mat = word & kAdjMat;
            }
            uint32_t left = __ballot_sync(0xFFFFFFFFu, mat != 0xFFFFFFFFu);
            while (left) {
                const uint32_t m = __shfl_sync(0xFFFFFFFFu, mat, __ffs(left) - 1);
                const bool mine = mat == m;
                float x = mine ? ga.x : 0.0f, y = mine ? ga.y : 0.0f, z = mine ? ga.z : 0.0f, w = mine ? gr : 0.0f;
                for (int off = 16; off; off >>= 1) {
                    x += __shfl_xor_sync(0xFFFFFFFFu, x, off);
                    y += __shfl_xor_sync(0xFFFFFFFFu, y, off);
                    z += __shfl_xor_sync(0xFFFFFFFFu, z, off);
                    w += __shfl_xor_sync(0xFFFFFFFFu, w, off);
                }
                if (lane < 4u) atomicAdd(&sm[4 * m + lane], lane == 0 ? x : (lane == 1 ? y : (lane == 2 ? z : w)));
                left &= ~__ballot_sync(0xFFFFFFFFu, mine);
            }
        }
    }
    __syncthreads();
    const uint32_t nm = min(P.num_mats, (uint32_t)kAdjMaxMats);
    for (uint32_t i = threadIdx.x; i < 4 * nm; i += blockDim.x) {
        if (sm[i] == 0.0f) continue;
        if ((i & 3u) < 3u)
            atomicAdd(&P.g_albedo[3 * (i >> 2) + (i & 3u)], sm[i]);
        else
            atomicAdd(&P.g_rough[i >> 2], sm[i]);
    }
}

// paths of a chunk at most, and the bytes its state and records may take (2^21
// paths of four bounces: 1.7 GB)
constexpr uint32_t kAdjStagePaths = 1u << 21;
constexpr size_t kAdjStageBytes = 4ull << 30;

// *done = false (nothing launched) where the one-thread-per-path kernels have
// to run: more pixels than a chunk holds or has room for, no memory
template <int ISECT>
static int run_staged(Context& C, const DevScene& S, const AdjParams& P, int mode, float* image, bool* done) {
    *done = false;
    const uint32_t npix = C.cam.w * C.cam.h;
    if (S.bounces == 0 || S.bounces > 1024) return NOOR_OK;
    if (!S.frames4 && !ref_words_fit(S.num_nodes)) return NOOR_OK;
    const bool record = mode == 1;
    const uint32_t verts = record ? S.bounces : 1u;
    // bytes a path takes below
    const size_t per_path = 180 + 48 * (size_t)verts + (record ? 100 * (size_t)verts + 4 : 16);
    const size_t most = std::min<size_t>(kAdjStagePaths, kAdjStageBytes / per_path);
    if (npix > most) return NOOR_OK;
    // samples a chunk, halved until the device has room and the context's limit allows
    uint32_t chunk = std::min<uint32_t>(P.spp, (uint32_t)(most / npix));
    size_t n, at, o, d, beta, L, hit, hit2, q0, q1, qs, qsh, sho, shd, pend, pbeta, ta, te, td, sc, vw, nv, lb, kh, cnt, first;
    auto place = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) & ~(size_t)255;
        return p;
    };
    for (;; chunk /= 2) {
        if (chunk == 0) return NOOR_OK;
        n = (size_t)npix * chunk;
        at = 0;
        o = place(16 * n), d = place(16 * n), beta = place(16 * n), L = place(16 * n), hit = place(16 * n);
        hit2 = place(8 * n), q0 = place(4 * n), q1 = place(4 * n), qs = place(4 * n * kStageKinds), qsh = place(8 * n);
        sho = place(32 * n), shd = place(32 * n), pend = place(32 * n * verts), pbeta = place(16 * n * verts);
        ta = place(record ? 32 * n * verts : 0), te = place(record ? 32 * n * verts : 0);
        td = place(record ? 16 * n * verts : 0), sc = place(record ? 16 * n * verts : 0);
        vw = place(record ? 4 * n * verts : 0), nv = place(record ? 4 * n : 0);
        lb = place(record ? 0 : 16 * n), kh = place(record ? 0 : 32 * (size_t)npix);
        cnt = place(4 * (size_t)kStWords * (S.bounces + 1)), first = place(16 * (size_t)chunk);
        if (at <= C.adj_bytes) break;
        if (at > C.workspace_limit) continue;
        if (C.adj_buf) cudaFree(C.adj_buf);
        C.adj_bytes = 0;
        if (cudaMalloc(&C.adj_buf, at) == cudaSuccess) {
            C.adj_bytes = at;
            break;
        }
        cudaGetLastError();
        C.adj_buf = nullptr;
    }
    char* p = static_cast<char*>(C.adj_buf);
    AdjStage A{};
    StageDev& W = A.W;
    W.o = (float4*)(p + o);
    W.d = (float4*)(p + d);
    W.beta = (float4*)(p + beta);
    W.L = (float4*)(p + L);
    W.hit = (float4*)(p + hit);
    W.hit2 = (uint2*)(p + hit2);
    W.queue[0] = (uint32_t*)(p + q0);
    W.queue[1] = (uint32_t*)(p + q1);
    W.qshade = (uint32_t*)(p + qs);
    W.qshadow = (uint32_t*)(p + qsh);
    W.sh_o = (float4*)(p + sho);
    W.sh_d = (float4*)(p + shd);
    W.pend = (float4*)(p + pend);
    W.pbeta = (float4*)(p + pbeta);
    W.count = (uint32_t*)(p + cnt);
    W.first = (float4*)(p + first);
    W.status = C.status;
    W.cap = (uint32_t)n;
    W.keep = record ? (uint32_t)n : 0u;
    if (record) {
        A.term_a = (float4*)(p + ta);
        A.term_e = (float4*)(p + te);
        A.term_d = (float2*)(p + td);
        A.scatter = (float4*)(p + sc);
        A.vertex = (uint32_t*)(p + vw);
        A.count = (uint32_t*)(p + nv);
    }
    float4* Lbuf = record ? nullptr : (float4*)(p + lb);
    constexpr int trav = 64;
    const size_t sm = (size_t)S.stack_words * trav * sizeof(uint32_t);
    cudaError_t e = allow_stacks(adj_trace<ISECT>, trav);
    if (e != cudaSuccess) return cuda_fail(e, "adjoint setup");
    for (uint32_t c0 = 0; c0 < P.spp; c0 += chunk) {
        W.frames = std::min(chunk, P.spp - c0);
        W.paths = npix * W.frames;
        W.frame0 = P.frame0 + c0;
        const uint32_t all = (W.paths + 255) / 256;
        const uint32_t gt = std::min<uint32_t>((W.paths + trav - 1) / trav, (uint32_t)C.sm_count * 16);
        const dim3 gs(std::min<uint32_t>((W.paths + 127) / 128, (uint32_t)C.sm_count * 8), kStageKinds);
        e = cudaMemsetAsync(W.count, 0, (char*)(W.first + W.frames) - (char*)W.count, C.stream);
        if (e != cudaSuccess) return cuda_fail(e, "adjoint");
        adj_begin<<<all, 256, 0, C.stream>>>(C.cam, A);
        adj_trace<ISECT><<<gt, trav, sm, C.stream>>>(S, C.cam, W, -1);
        C.launches += 4;
        for (uint32_t b = 0; b < S.bounces; ++b) {
            // every path may have ended long before the limit (kStageAsk)
            if (b && b % kStageAsk == 0 && S.bounces - b >= kStageAsk) {
                uint32_t left = 0;
                if ((e = cudaMemcpyAsync(&left, W.count + b * kStWords + kStActive, 4, cudaMemcpyDeviceToHost,
                                         C.stream)) ||
                    (e = cudaStreamSynchronize(C.stream)))
                    return cuda_fail(e, "adjoint");
                if (left == 0) break;
            }
            C.launches += 2;
            if (record)
                adj_shade<ISECT, true><<<gs, 128, 0, C.stream>>>(S, P, A, b);
            else
                adj_shade<ISECT, false><<<gs, 128, 0, C.stream>>>(S, P, A, b);
            adj_trace<ISECT><<<dim3(gt, 2), trav, sm, C.stream>>>(S, C.cam, W, (int)b);
        }
        adj_finish<ISECT><<<all, 256, 0, C.stream>>>(S, C.cam, P, A, Lbuf);
        if (record)
            adj_backprop<<<std::min<uint32_t>((W.paths + kAdjBlock - 1) / kAdjBlock, (uint32_t)C.sm_count * 12), kAdjBlock,
                           0, C.stream>>>(S, C.cam, P, A);
        else
            adjoint_accumulate(npix, W.frames, Lbuf, (float4*)(p + kh), c0 == 0, c0 + W.frames >= P.spp,
                               1.0f / (float)P.spp, image, C.stream);
        e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "adjoint");
    }
    *done = true;
    return sync_and_check(C, "adjoint");
}

int adjoint_staged(Context& C, const DevScene& S, const AdjParams& P, int mode, float* image, bool* done) {
    return S.isect == NOOR_ISECT_WATERTIGHT ? run_staged<NOOR_ISECT_WATERTIGHT>(C, S, P, mode, image, done)
                                            : run_staged<NOOR_ISECT_REF_WALD>(C, S, P, mode, image, done);
}

}  // namespace nb
