// What the adjoint's two forms share: parameters, BSDF values with their
// derivatives, environment texels, the estimator's terms.
#pragma once
#include "integrator.cuh"
#include "runtime.h"

namespace nb {

struct AdjParams {
    const float* albedo;     // M x 3
    const float* rough;      // M
    const float* env;        // H x W x 3 (radiance texels for evaluation)
    int env_w, env_h;
    float* g_albedo;         // M x 3
    float* g_rough;          // M
    float* g_env;            // H x W x 3
    const float* grad_img;   // npix x 3
    float* image;            // npix x 3
    uint32_t num_mats;
    uint32_t spp;
    uint32_t frame0;
    uint32_t* status;
};

// material with the evaluation parameters substituted
NB_D DevMaterial eval_material(const DevMaterial& m0, const AdjParams& P, uint32_t mi) {
    DevMaterial m = m0;
    const float3 a = f3(P.albedo[3 * mi], P.albedo[3 * mi + 1], P.albedo[3 * mi + 2]);
    if (lobe_of(m.type) == kLobeLambert) m.diffuse = a;
    if (lobe_of(m.type) == kLobeConductor) {
        m.specular = a;
        m.rough_x = m.rough_y = P.rough[mi];
    }
    return m;
}

// f, the value without the tint (conductor), and dlog f / droughness
struct FDeriv {
    float3 f;
    float3 f_untinted;
    float dlogf_dr;
};

NB_D float ggx_dlogD_dalpha(const float3& wh, float a) {
    const float t2 = tan2t(wh);
    if (isinf(t2)) return 0.0f;
    const float a2 = a * a;
    return 2.0f * (t2 - a2) / (a * (a2 + t2));
}
NB_D float ggx_dlambda_dalpha(const float3& w, float a) {
    const float at = fabsf(tant(w));
    if (isinf(at)) return 0.0f;
    const float t2 = at * at;
    return a * t2 / (2.0f * sqrtf(1.0f + a * a * t2));
}
// Beckmann: D = exp(-tan^2/a^2) / (pi a^2 cos^4); Lambda is the rational fit
// in x = 1 / (a |tan|), zero for x >= 1.6
NB_D float beck_dlogD_dalpha(const float3& wh, float a) {
    const float t2 = tan2t(wh);
    if (isinf(t2)) return 0.0f;
    return 2.0f * t2 / (a * a * a) - 2.0f / a;
}
NB_D float beck_dlambda_dalpha(const float3& w, float a) {
    const float at = fabsf(tant(w));
    if (isinf(at)) return 0.0f;
    const float x = 1.0f / (a * at);
    if (x >= 1.6f) return 0.0f;
    const float n = 1.0f - 1.259f * x + 0.396f * x * x, dn = -1.259f + 0.792f * x;
    const float q = 3.535f * x + 2.181f * x * x, dq = 3.535f + 4.362f * x;
    const float dlam_dx = (dn * q - n * dq) / (q * q);
    return dlam_dx * (-x / a);
}

// BSDF value at (wo, wi) in the local frame with the evaluation material
NB_D FDeriv lobe_value(uint32_t lobe, const DevMaterial& m, const Frame& F, const float3& woW, const float3& wiW) {
    FDeriv r{f3(0.0f), f3(0.0f), 0.0f};
    const float3 wo = to_local_o(F, woW), wi = to_local_i(F, wiW);
    const bool reflect = dot(wiW, F.ng) * dot(woW, F.ng) > 0.0f;
    if (!reflect) return r;
    if (lobe == kLobeLambert) {
        r.f = m.diffuse * kInvPi;
        r.f_untinted = f3(kInvPi);
        return r;
    }
    if (lobe == kLobeConductor) {
        if (!same_hemi(wo, wi)) return r;
        const float cO = fabsf(wo.z), cI = fabsf(wi.z);
        if (cI == 0.0f || cO == 0.0f) return r;
        float3 wh = normalize_fast(wi + wo);
        if (is_black(wh)) return r;
        wh *= signf_ref(wh.z);
        const float3 Fr = fresnel_conductor(dot(wo, wh), m.ior, m.k);
        const Micro mf = make_micro(m);
        const float D = mf.D(wh), G = mf.G(wo, wi);
        r.f_untinted = Fr * D * G / (4.0f * cI * cO);
        r.f = r.f_untinted * m.specular;
        const float a = mf.ax;
        const float r2 = m.rough_x * m.rough_x;
        // alpha = max(r^2, 1e-3): dalpha/dr = 2r above the floor, 0 on it
        if (r2 > 1e-3f) {
            const float dla = mf.dist == 0u ? ggx_dlogD_dalpha(wh, a) -
                                                  (ggx_dlambda_dalpha(wo, a) + ggx_dlambda_dalpha(wi, a)) * G
                                            : beck_dlogD_dalpha(wh, a) -
                                                  (beck_dlambda_dalpha(wo, a) + beck_dlambda_dalpha(wi, a)) * G;
            r.dlogf_dr = dla * 2.0f * m.rough_x;
        }
    }
    return r;
}

// bilinear texel weights of direction `dir` in the evaluation env map
struct Bilerp {
    int idx[4];
    float w[4];
};
NB_D Bilerp env_weights(const AdjParams& P, const float3& dir) {
    const float u = spherical_phi(dir) * kInv2Pi, v = spherical_theta(dir) * kInvPi;
    const int W = P.env_w, H = P.env_h;
    const float x = u * (float)W - 0.5f, y = v * (float)H - 0.5f;
    const float fx0 = floorf(x), fy0 = floorf(y);
    const float ax = x - fx0, ay = y - fy0;
    int x0 = (int)fx0, y0 = (int)fy0, x1 = x0 + 1, y1 = y0 + 1;
    x0 = min(max(x0, 0), W - 1);
    x1 = min(max(x1, 0), W - 1);
    y0 = min(max(y0, 0), H - 1);
    y1 = min(max(y1, 0), H - 1);
    Bilerp b;
    b.idx[0] = y0 * W + x0;
    b.idx[1] = y0 * W + x1;
    b.idx[2] = y1 * W + x0;
    b.idx[3] = y1 * W + x1;
    b.w[0] = (1.0f - ax) * (1.0f - ay);
    b.w[1] = ax * (1.0f - ay);
    b.w[2] = (1.0f - ax) * ay;
    b.w[3] = ax * ay;
    return b;
}
NB_D float3 env_radiance(const AdjParams& P, const Bilerp& b) {
    float3 c = f3(0.0f);
    for (int k = 0; k < 4; ++k)
        c += b.w[k] * f3(P.env[3 * b.idx[k]], P.env[3 * b.idx[k] + 1], P.env[3 * b.idx[k] + 2]);
    return c;
}

// One term X (.) f * s of the estimator: X is light radiance (env texels
// when `env`), f the BSDF value at the vertex.
struct Term {
    float3 X;
    FDeriv f;
    float s;
    bool env;
    Bilerp bl;
    float xscale;   // light-count factor multiplying the env radiance
};

constexpr int kAdjBlock = 128;
constexpr int kAdjMaxMats = 256;
// The staged form (adjoint_stages.cu).  *done = false, and nothing launched,
// where the kernels with a thread per path have to run.
int adjoint_staged(Context& C, const DevScene& S, const AdjParams& P, int mode, float* image, bool* done);
void adjoint_accumulate(uint32_t npix, uint32_t nc, const float4* Lbuf, float4* kahan, int first, int last, float inv_spp,
                        float* image, cudaStream_t s);

}  // namespace nb
