// Two-level BVH traversal (closest hit and any hit) with a per-thread stack
// in shared memory, and the two ray/triangle tests:
//   * NOOR_ISECT_REF_WALD: the reference's Wald projection test
//     (noor/cuda/triangle.cuh:82-198), evaluated with exactly rounded
//     operations in the order the source writes them;
//   * NOOR_ISECT_WATERTIGHT: Woop, Benthin & Wald 2013, "Watertight
//     Ray/Triangle Intersection" (JCGT 2(1)), with its double-precision
//     fallback on zero edge functions.
// The traversal order reproduces noor/cuda/bvh.cuh:142-234: pop, slab test,
// then by node kind; an inner node pushes the far child first so the near
// child (chosen by the ray's direction sign on the split axis) pops next.
#pragma once
#include "scene_dev.cuh"
#include "wide_bvh.h"

namespace nb {

// ray in the space of the BVH level being traversed
struct TRay {
    float3 o, d, inv;
    uint32_t neg;  // bit a set when d[a] <= 0 (noor/cuda/ray.cuh:200-206)
};

NB_D void tray_setup(TRay& r, const float3& o, const float3& d) {
    r.o = o;
    r.d = d;
    r.inv = f3(xdiv(1.0f, d.x), xdiv(1.0f, d.y), xdiv(1.0f, d.z));
    r.neg = (d.x > 0.0f ? 0u : 1u) | (d.y > 0.0f ? 0u : 2u) | (d.z > 0.0f ? 0u : 4u);
}

// world -> object: origin as translation + M*o, direction as M*d, no
// renormalisation, so t is shared by both levels (noor/cuda/ray.cuh:174-180)
NB_D void tray_to_object(TRay& r, const TRay& w, const DevXform* xf) {
    const float4 r0 = __ldg(&xf->w2o[0]);
    const float4 r1 = __ldg(&xf->w2o[1]);
    const float4 r2 = __ldg(&xf->w2o[2]);
    const float3 o = f3(xadd(r0.w, xdot3(r0.x, r0.y, r0.z, w.o.x, w.o.y, w.o.z)),
                        xadd(r1.w, xdot3(r1.x, r1.y, r1.z, w.o.x, w.o.y, w.o.z)),
                        xadd(r2.w, xdot3(r2.x, r2.y, r2.z, w.o.x, w.o.y, w.o.z)));
    const float3 d = f3(xdot3(r0.x, r0.y, r0.z, w.d.x, w.d.y, w.d.z),
                        xdot3(r1.x, r1.y, r1.z, w.d.x, w.d.y, w.d.z),
                        xdot3(r2.x, r2.y, r2.z, w.d.x, w.d.y, w.d.z));
    tray_setup(r, o, d);
}

// A ray whose origin and direction components are all finite and non-zero:
// an identity transform maps it onto itself bit for bit (1 x = x, 0 y = +-0,
// x +- 0 = x), which a zero or non-finite component would not guarantee
// (-0 turns into +0, 0 inf into NaN).
NB_D bool ray_plain(const float3& o, const float3& d) {
    const float m = 3.40282347e38f;
    const float ao[3] = {fabsf(o.x), fabsf(o.y), fabsf(o.z)}, ad[3] = {fabsf(d.x), fabsf(d.y), fabsf(d.z)};
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) ok = ok && ao[i] > 0.0f && ao[i] <= m && ad[i] > 0.0f && ad[i] <= m;
    return ok;
}

// The level's ray moved into instance `ins`'s object space
// (noor/cuda/ray.cuh:174-180).  An instance whose world-to-object rows are
// exactly the identity (DevScene::xf_ident, set at upload) leaves a plain
// ray as it is, so the world ray is kept.  Returns whether the level's ray
// is the world ray.
NB_D bool enter_instance(TRay& lr, const TRay& wr, const DevScene& S, uint32_t ins, bool plain) {
    if (plain && ((__ldg(&S.xf_ident[ins >> 5]) >> (ins & 31u)) & 1u)) {
        lr = wr;
        return true;
    }
    tray_to_object(lr, wr, S.xforms + ins);
    return false;
}

// slab test of noor/cuda/bbox.cuh:62-80
template <class Ray>
NB_D bool slab_hit_f(const Ray& r, float mnx, float mny, float mnz, float mxx, float mxy, float mxz, float tmax) {
    const bool nx = r.neg & 1u, ny = r.neg & 2u, nz = r.neg & 4u;
    float tMin = xmul(xsub(nx ? mxx : mnx, r.o.x), r.inv.x);
    float tMax = xmul(xsub(nx ? mnx : mxx, r.o.x), r.inv.x);
    const float tyMin = xmul(xsub(ny ? mxy : mny, r.o.y), r.inv.y);
    const float tyMax = xmul(xsub(ny ? mny : mxy, r.o.y), r.inv.y);
    if (tMin > tyMax || tyMin > tMax) return false;
    if (tyMin > tMin) tMin = tyMin;
    if (tyMax < tMax) tMax = tyMax;
    const float tzMin = xmul(xsub(nz ? mxz : mnz, r.o.z), r.inv.z);
    const float tzMax = xmul(xsub(nz ? mnz : mxz, r.o.z), r.inv.z);
    if (tMin > tzMax || tzMin > tMax) return false;
    if (tzMin > tMin) tMin = tzMin;
    if (tzMax < tMax) tMax = tzMax;
    return (tMin < tmax) && (tMax > 0.0f);
}
template <class Ray>
NB_D bool slab_hit(const Ray& r, const uint4& lo, const uint4& hi, float tmax) {
    return slab_hit_f(r, __uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z), __uint_as_float(hi.x),
                      __uint_as_float(hi.y), __uint_as_float(hi.z), tmax);
}

// Wald projection test (noor/cuda/triangle.cuh:82-141); on success writes
// t into tmax and the barycentrics (u weights v1, v weights v2).
template <class Ray>
NB_D bool wald_test(const Ray& r, const DevWaldTri* tri, float& tmax, float& bu, float& bv,
                    uint32_t& mtype) {
    const uint4 a = __ldg(&tri->ax_nu_nv_nd);
    const uint4 c = __ldg(&tri->cnu_cnv_deg_mat);
    if (c.z == 1u) return false;
    const uint32_t k = a.x;
    const uint32_t ku = (k == 0u) ? 1u : (k == 1u ? 2u : 0u);
    const uint32_t kv = (k == 0u) ? 2u : (k == 1u ? 0u : 1u);
    const float ro_u = comp(r.o, ku), ro_v = comp(r.o, kv), ro_k = comp(r.o, k);
    const float rd_u = comp(r.d, ku), rd_v = comp(r.d, kv), rd_k = comp(r.d, k);
    const float nu = __uint_as_float(a.y), nv = __uint_as_float(a.z), nd = __uint_as_float(a.w);
    const float denom = xadd(xadd(rd_k, xmul(nu, rd_u)), xmul(nv, rd_v));
    if (denom == 0.0f) return false;
    const float t = xdiv(xsub(xsub(xsub(nd, ro_k), xmul(nu, ro_u)), xmul(nv, ro_v)), denom);
    if (t < 0.0f || t > tmax) return false;
    const uint4 b = __ldg(&tri->bnu_bnv_au_av);
    const float hu = xsub(xadd(ro_u, xmul(t, rd_u)), __uint_as_float(b.z));
    const float hv = xsub(xadd(ro_v, xmul(t, rd_v)), __uint_as_float(b.w));
    const float u = xadd(xmul(hv, __uint_as_float(b.x)), xmul(hu, __uint_as_float(b.y)));
    const float v = xadd(xmul(hu, __uint_as_float(c.x)), xmul(hv, __uint_as_float(c.y)));
    if (!(u >= 0.0f && v >= 0.0f && xadd(u, v) <= 1.0f)) return false;
    tmax = t;
    bu = u;
    bv = v;
    mtype = c.w;
    return true;
}

// per-ray constants of the watertight test
struct WtRay {
    int kx, ky, kz;
    float sx, sy, sz;
};

NB_D void wt_setup(WtRay& w, const float3& d) {
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz + 1 == 3 ? 0 : kz + 1;
    int ky = kx + 1 == 3 ? 0 : kx + 1;
    const float dz = comp(d, kz);
    if (dz < 0.0f) {
        const int t = kx;
        kx = ky;
        ky = t;
    }
    w.kx = kx;
    w.ky = ky;
    w.kz = kz;
    w.sx = xdiv(comp(d, kx), dz);
    w.sy = xdiv(comp(d, ky), dz);
    w.sz = xdiv(1.0f, dz);
}

NB_D float xorsign(float v, uint32_t signbit) { return __uint_as_float(__float_as_uint(v) ^ signbit); }

template <class Ray>
NB_D bool wt_test(const Ray& r, const WtRay& w, const DevWtTri* tri, float& tmax, float& bu,
                  float& bv, uint32_t& mtype) {
    const float4 p0 = __ldg(&tri->v0);
    const float4 p1 = __ldg(&tri->v1);
    const float4 p2 = __ldg(&tri->v2);
    const float3 A = f3(xsub(p0.x, r.o.x), xsub(p0.y, r.o.y), xsub(p0.z, r.o.z));
    const float3 B = f3(xsub(p1.x, r.o.x), xsub(p1.y, r.o.y), xsub(p1.z, r.o.z));
    const float3 C = f3(xsub(p2.x, r.o.x), xsub(p2.y, r.o.y), xsub(p2.z, r.o.z));
    const float Akz = comp(A, w.kz), Bkz = comp(B, w.kz), Ckz = comp(C, w.kz);
    const float Ax = xsub(comp(A, w.kx), xmul(w.sx, Akz));
    const float Ay = xsub(comp(A, w.ky), xmul(w.sy, Akz));
    const float Bx = xsub(comp(B, w.kx), xmul(w.sx, Bkz));
    const float By = xsub(comp(B, w.ky), xmul(w.sy, Bkz));
    const float Cx = xsub(comp(C, w.kx), xmul(w.sx, Ckz));
    const float Cy = xsub(comp(C, w.ky), xmul(w.sy, Ckz));
    float U = xsub(xmul(Cx, By), xmul(Cy, Bx));
    float V = xsub(xmul(Ax, Cy), xmul(Ay, Cx));
    float W = xsub(xmul(Bx, Ay), xmul(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        // products of two floats are exact in double; one rounding each
        U = (float)__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx));
        V = (float)__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx));
        W = (float)__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax));
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = xadd(xadd(U, V), W);
    if (det == 0.0f) return false;
    const float Az = xmul(w.sz, Akz), Bz = xmul(w.sz, Bkz), Cz = xmul(w.sz, Ckz);
    const float T = xadd(xadd(xmul(U, Az), xmul(V, Bz)), xmul(W, Cz));
    const uint32_t sgn = __float_as_uint(det) & 0x80000000u;
    const float Ts = xorsign(T, sgn);
    if (Ts < 0.0f || Ts > xmul(tmax, xorsign(det, sgn))) return false;
    const float rcp = xdiv(1.0f, det);
    tmax = xmul(T, rcp);
    bu = xmul(V, rcp);
    bv = xmul(W, rcp);
    mtype = __float_as_uint(p0.w);
    return true;
}

// The alpha cut of an ALPHA material's triangle (noor/cuda/triangle.cuh:
// 124-133): the transparency map at the hit's interpolated uv; a texel of
// 1e-4 or less lets the ray through.
template <int ISECT>
NB_OUTLINE bool alpha_cut(const DevScene& S, uint32_t ti, float bu, float bv) {
    const uint4 a = ISECT == NOOR_ISECT_WATERTIGHT ? __ldg(&S.wtri[ti].attr) : __ldg(&S.wald[ti].attr);
    const float2 uv = lerp_uv(vertex_uv(S, a.x), vertex_uv(S, a.y), vertex_uv(S, a.z), bu, bv);
    return slot_tex(S.mat_tex[a.w], kTexAlpha, uv).x <= 0.0001f;
}

// Arithmetic of the light-shape tests: with X (the reference's Wald mode,
// whose hit distances are the reference's to the bit) each operation rounds
// on its own; otherwise the compiler may contract multiply-adds.
template <bool X> NB_D float smul(float a, float b) { return X ? __fmul_rn(a, b) : a * b; }
template <bool X> NB_D float sadd(float a, float b) { return X ? __fadd_rn(a, b) : a + b; }
template <bool X> NB_D float ssub(float a, float b) { return X ? __fsub_rn(a, b) : a - b; }
template <bool X> NB_D float sdot(float ax, float ay, float az, float bx, float by, float bz) {
    return sadd<X>(sadd<X>(smul<X>(ax, bx), smul<X>(ay, by)), smul<X>(az, bz));
}

// quad of an area light (noor/cuda/geometry.cuh:105-123); note the
// reference accepts negative t (no lower bound), kept as is.
template <bool X = false>
NB_D bool quad_hit(const DevAreaLight& q, const float3& o, const float3& d, float& tmax) {
    const float denom = sdot<X>(q.n.x, q.n.y, q.n.z, d.x, d.y, d.z);
    if (denom == 0.0f) return false;
    const float t = -ssub<X>(sdot<X>(o.x, o.y, o.z, q.n.x, q.n.y, q.n.z),
                             sdot<X>(q.center.x, q.center.y, q.center.z, q.n.x, q.n.y, q.n.z)) /
                    denom;
    if (t > tmax) return false;
    // pointAtParameter(t) - center
    const float ix = ssub<X>(sadd<X>(o.x, smul<X>(t, d.x)), q.center.x);
    const float iy = ssub<X>(sadd<X>(o.y, smul<X>(t, d.y)), q.center.y);
    const float iz = ssub<X>(sadd<X>(o.z, smul<X>(t, d.z)), q.center.z);
    const float t0 = sdot<X>(ix, iy, iz, q.u.x, q.u.y, q.u.z) / sdot<X>(q.u.x, q.u.y, q.u.z, q.u.x, q.u.y, q.u.z);
    if (t0 < 0.0f || t0 > 1.0f) return false;
    const float t1 = sdot<X>(ix, iy, iz, q.v.x, q.v.y, q.v.z) / sdot<X>(q.v.x, q.v.y, q.v.z, q.v.x, q.v.y, q.v.z);
    if (t1 < 0.0f || t1 > 1.0f) return false;
    tmax = t;
    return true;
}

// solveQuadratic (noor/cuda/utils.cuh:52-91): the root of larger magnitude
// first, the other from x0 * x1 = c / a; returns x0 <= x1
template <bool X = false>
NB_D bool solve_quadratic(float a, float b, float c, float& x0, float& x1) {
    if (a == 0.0f) {
        if (b != 0.0f) {
            x0 = x1 = -c / b;
            return true;
        }
        return false;
    }
    const float disc = ssub<X>(smul<X>(b, b), smul<X>(smul<X>(4.0f, a), c));
    if (disc < 0.0f) return false;
    const float sd = sqrtf(disc);
    const float q = b < 0.0f ? smul<X>(-0.5f, ssub<X>(b, sd)) : smul<X>(-0.5f, sadd<X>(b, sd));
    x0 = q / a;
    x1 = c / q;
    if (x0 > x1) {
        const float t = x0;
        x0 = x1;
        x1 = t;
    }
    return true;
}

// sphere of an area light (noor/cuda/geometry.cuh:125-150): nearest root in
// [0, tmax], else the far root when the near one is behind the origin
template <bool X = false>
NB_D bool sphere_hit(const DevAreaLight& s, const float3& o, const float3& d, float& tmax) {
    const float ox = ssub<X>(o.x, s.center.x), oy = ssub<X>(o.y, s.center.y), oz = ssub<X>(o.z, s.center.z);
    float t0, t1;
    if (!solve_quadratic<X>(sdot<X>(d.x, d.y, d.z, d.x, d.y, d.z), smul<X>(2.0f, sdot<X>(ox, oy, oz, d.x, d.y, d.z)),
                            ssub<X>(sdot<X>(ox, oy, oz, ox, oy, oz), s.radius2), t0, t1))
        return false;
    if (!(t0 <= tmax && t1 >= 0.0f)) return false;
    if (t0 < 0.0f) {
        if (t1 > tmax) return false;
        tmax = t1;
    } else {
        tmax = t0;
    }
    return true;
}

// disk of an area light (noor/cuda/geometry.cuh:152-163); like the quad, no
// lower bound on t
template <bool X = false>
NB_D bool disk_hit(const DevAreaLight& q, const float3& o, const float3& d, float& tmax) {
    const float denom = sdot<X>(q.n.x, q.n.y, q.n.z, d.x, d.y, d.z);
    if (denom == 0.0f) return false;
    const float t = -ssub<X>(sdot<X>(o.x, o.y, o.z, q.n.x, q.n.y, q.n.z),
                             sdot<X>(q.center.x, q.center.y, q.center.z, q.n.x, q.n.y, q.n.z)) /
                    denom;
    if (t > tmax) return false;
    const float px = ssub<X>(sadd<X>(o.x, smul<X>(t, d.x)), q.center.x);
    const float py = ssub<X>(sadd<X>(o.y, smul<X>(t, d.y)), q.center.y);
    const float pz = ssub<X>(sadd<X>(o.z, smul<X>(t, d.z)), q.center.z);
    if (sdot<X>(px, py, pz, px, py, pz) > q.radius2) return false;
    tmax = t;
    return true;
}

// CudaShape::intersect (noor/cuda/shapeimp.cuh:73-87).  EXT false: the
// scene's area lights are all quads (kernels for such scenes leave the
// other shapes' code out)
template <bool EXT = true, bool X = false>
NB_D bool shape_hit(const DevAreaLight& a, const float3& o, const float3& d, float& tmax) {
    if (!EXT || a.type == NOOR_SHAPE_QUAD) return quad_hit<X>(a, o, d, tmax);
    if (a.type == NOOR_SHAPE_SPHERE) return sphere_hit<X>(a, o, d, tmax);
    return disk_hit<X>(a, o, d, tmax);
}

struct HitRec {
    float u, v;
    uint32_t tri;
    uint32_t ins;
    uint32_t mtype;
};

// Shared-memory stack: entry i of this thread lives at stk[i * stride].
struct SmemStack {
    uint32_t* base;
    int stride;
    int cap;
};

// Node kinds that are not inner nodes (an inner node has none of these bits)
constexpr uint32_t kNodeKindMask =
    NOOR_LIGHT_NODE_MASK | NOOR_MESH_INSTANCE_MASK | NOOR_MESH_LEAF_MASK | NOOR_TRI_LEAF_MASK;
constexpr uint32_t kNoNode = 0xFFFFFFFFu;

// Closest hit.  tmax in: ray extent, out: hit distance.  Returns hit flag;
// on stack overflow sets *status and returns what was found so far.
// The visit order is that of the reference's stack loop: the node the
// reference would pop next (the near child of an inner node, the last child
// of a mesh leaf, the root of an instance) is kept in a register instead of
// being pushed and popped at once, and inner nodes are dispatched first.
template <int ISECT, bool EXT = true>
NB_D bool trace_closest(const DevScene& S, const float3& o, const float3& d, float& tmax,
                        HitRec& rec, const SmemStack& st, uint32_t* status) {
    TRay wr;
    tray_setup(wr, o, d);
    TRay lr = wr;
    WtRay wt;
    if (ISECT == NOOR_ISECT_WATERTIGHT) wt_setup(wt, lr.d);
    bool wtw = true;  // wt holds the world ray's constants
    const bool plain = ray_plain(o, d);
    float ltmax = tmax;
    uint32_t ins = 0;
    bool hit = false;
    int top = 0;
    uint32_t ni = S.root;
    for (;;) {
        const DevNode* nd = S.nodes + ni;
        const uint4 lo = __ldg(&nd->lo);
        const uint4 hi = __ldg(&nd->hi);
        uint32_t next = kNoNode;
        if (hi.w & NOOR_MESH_NODE_MASK) {
            lr = wr;
            ltmax = tmax;
            if (ISECT == NOOR_ISECT_WATERTIGHT && !wtw) {
                wt_setup(wt, wr.d);
                wtw = true;
            }
        }
        if (slab_hit(lr, lo, hi, ltmax)) {
            if (!(hi.w & kNodeKindMask)) {
                // inner: the near child (by the ray's sign on the split axis) next, the far one pushed
                if (top + 1 > st.cap) { atomicOr(status, NOOR_DEV_STACK_OVERFLOW); break; }
                const uint32_t axis = hi.w & NOOR_AXIS_MASK;
                const bool neg = (lr.neg >> axis) & 1u;
                st.base[top * st.stride] = neg ? ni + 1 : lo.w;
                ++top;
                next = neg ? lo.w : ni + 1;
            } else if (hi.w & NOOR_LIGHT_NODE_MASK) {
                const uint32_t li = hi.w & NOOR_LIGHT_MASK;
                if ((int)li < S.num_area_lights &&
                    shape_hit<EXT, ISECT == NOOR_ISECT_REF_WALD>(S.area_lights[li], o, d, tmax)) {
                    hit = true;
                    rec.ins = li;
                    rec.mtype = NOOR_MESHLIGHT | NOOR_EMITTER;
                }
            } else if (hi.w & NOOR_MESH_INSTANCE_MASK) {
                ins = hi.w & NOOR_TRANS_MASK;
                const bool same = enter_instance(lr, wr, S, ins, plain);
                ltmax = tmax;
                if (ISECT == NOOR_ISECT_WATERTIGHT && !(same && wtw)) {
                    wt_setup(wt, lr.d);
                    wtw = same;
                }
                next = lo.w;
            } else if (hi.w & NOOR_MESH_LEAF_MASK) {
                const uint32_t cnt = hi.w & NOOR_COUNT_MASK;
                if (top + (int)cnt > st.cap + 1) { atomicOr(status, NOOR_DEV_STACK_OVERFLOW); break; }
                for (uint32_t i = 1; i < cnt; ++i) {
                    st.base[top * st.stride] = ni + i;
                    ++top;
                }
                if (cnt) next = ni + cnt;
            } else {
                const uint32_t start = lo.w;
                const uint32_t end = start + (hi.w & NOOR_TRI_COUNT_MASK);
                bool leaf_hit = false;
                for (uint32_t ti = start; ti < end; ++ti) {
                    float bu, bv;
                    uint32_t mt;
                    bool h;
                    if (EXT && S.has_alpha) {
                        // the hit distance is kept only past the alpha cut
                        float tc = ltmax;
                        if (ISECT == NOOR_ISECT_WATERTIGHT)
                            h = wt_test(lr, wt, S.wtri + ti, tc, bu, bv, mt);
                        else
                            h = wald_test(lr, S.wald + ti, tc, bu, bv, mt);
                        if (h && (mt & NOOR_ALPHA) && alpha_cut<ISECT>(S, ti, bu, bv)) h = false;
                        if (h) ltmax = tc;
                    } else if (ISECT == NOOR_ISECT_WATERTIGHT) {
                        h = wt_test(lr, wt, S.wtri + ti, ltmax, bu, bv, mt);
                    } else {
                        h = wald_test(lr, S.wald + ti, ltmax, bu, bv, mt);
                    }
                    if (h) {
                        leaf_hit = true;
                        rec.u = bu;
                        rec.v = bv;
                        rec.tri = ti;
                        rec.mtype = mt;
                    }
                }
                if (leaf_hit) {
                    hit = true;
                    tmax = ltmax;
                    rec.ins = ins;
                }
            }
        }
        if (next == kNoNode) {
            if (top == 0) break;
            --top;
            next = st.base[top * st.stride];
        }
        ni = next;
    }
    return hit;
}

// Any hit within (0, tmax]; light nodes count as occluders.  Same visit
// order and register-held next node as trace_closest.
template <int ISECT, bool EXT = true>
NB_D bool trace_any(const DevScene& S, const float3& o, const float3& d, float tmax,
                    const SmemStack& st, uint32_t* status) {
    TRay wr;
    tray_setup(wr, o, d);
    TRay lr = wr;
    WtRay wt;
    if (ISECT == NOOR_ISECT_WATERTIGHT) wt_setup(wt, lr.d);
    bool wtw = true;  // wt holds the world ray's constants
    const bool plain = ray_plain(o, d);
    float ltmax = tmax;
    int top = 0;
    uint32_t ni = S.root;
    for (;;) {
        const DevNode* nd = S.nodes + ni;
        const uint4 lo = __ldg(&nd->lo);
        const uint4 hi = __ldg(&nd->hi);
        uint32_t next = kNoNode;
        if (hi.w & NOOR_MESH_NODE_MASK) {
            lr = wr;
            ltmax = tmax;
            if (ISECT == NOOR_ISECT_WATERTIGHT && !wtw) {
                wt_setup(wt, wr.d);
                wtw = true;
            }
        }
        if (slab_hit(lr, lo, hi, ltmax)) {
            if (!(hi.w & kNodeKindMask)) {
                if (top + 1 > st.cap) { atomicOr(status, NOOR_DEV_STACK_OVERFLOW); return false; }
                const uint32_t axis = hi.w & NOOR_AXIS_MASK;
                const bool neg = (lr.neg >> axis) & 1u;
                st.base[top * st.stride] = neg ? ni + 1 : lo.w;
                ++top;
                next = neg ? lo.w : ni + 1;
            } else if (hi.w & NOOR_LIGHT_NODE_MASK) {
                const uint32_t li = hi.w & NOOR_LIGHT_MASK;
                float tm = tmax;
                if ((int)li < S.num_area_lights && shape_hit<EXT, ISECT == NOOR_ISECT_REF_WALD>(S.area_lights[li], o, d, tm))
                    return true;
            } else if (hi.w & NOOR_MESH_INSTANCE_MASK) {
                const bool same = enter_instance(lr, wr, S, hi.w & NOOR_TRANS_MASK, plain);
                ltmax = tmax;
                if (ISECT == NOOR_ISECT_WATERTIGHT && !(same && wtw)) {
                    wt_setup(wt, lr.d);
                    wtw = same;
                }
                next = lo.w;
            } else if (hi.w & NOOR_MESH_LEAF_MASK) {
                const uint32_t cnt = hi.w & NOOR_COUNT_MASK;
                if (top + (int)cnt > st.cap + 1) { atomicOr(status, NOOR_DEV_STACK_OVERFLOW); return false; }
                for (uint32_t i = 1; i < cnt; ++i) {
                    st.base[top * st.stride] = ni + i;
                    ++top;
                }
                if (cnt) next = ni + cnt;
            } else {
                const uint32_t start = lo.w;
                const uint32_t end = start + (hi.w & NOOR_TRI_COUNT_MASK);
                for (uint32_t ti = start; ti < end; ++ti) {
                    float tm = ltmax, bu, bv;
                    uint32_t mt;
                    bool h;
                    if (ISECT == NOOR_ISECT_WATERTIGHT)
                        h = wt_test(lr, wt, S.wtri + ti, tm, bu, bv, mt);
                    else
                        h = wald_test(lr, S.wald + ti, tm, bu, bv, mt);
                    if (h && EXT && S.has_alpha && (mt & NOOR_ALPHA) && alpha_cut<ISECT>(S, ti, bu, bv)) h = false;
                    if (h) return true;
                }
            }
        }
        if (next == kNoNode) {
            if (top == 0) break;
            --top;
            next = st.base[top * st.stride];
        }
        ni = next;
    }
    return false;
}

// A ray below which the four-wide tree's boxes may not stand in for the
// binary tree's: a direction component that is zero or so small (or an origin
// or direction so large) that the box test's products could leave the range
// its error bound covers, or a component that is not a number.  Such rays
// walk the binary tree node by node.
NB_D bool wide_degenerate(const float3& o, const float3& d) {
    const float lo = 1e-18f, hi = 1e18f, far = kWideMaxCoord;
    const float3 a = f3(fabsf(d.x), fabsf(d.y), fabsf(d.z));
    return !(a.x >= lo && a.y >= lo && a.z >= lo && a.x <= hi && a.y <= hi && a.z <= hi && fabsf(o.x) <= far &&
             fabsf(o.y) <= far && fabsf(o.z) <= far);
}

// The level's ray as the wide nodes' box test takes it: a plane at x (on axis
// a) is met at x * inv[a] + c, c = -o[a] * inv[a] moved down (cn, near
// planes) or up (cf, far planes) by pad * |inv[a]|, which bounds what rounding
// adds: in units of the box coordinates, with u = 2^-24 and |x| <= reach, c
// and x * inv + c round at most u (2 |o| + reach), the exact slab test
// (x - o) * inv at most u * 2 (|o| + reach), in all below pad = 5 u (|o| +
// reach).
template <int ISECT>
struct BoxRay {
    float3 o, inv, cn, cf;
    uint32_t neg;       // bit a set when d[a] <= 0
};
template <>
struct BoxRay<NOOR_ISECT_REF_WALD> {
    float3 o, inv, cn, cf;
    uint32_t neg;
    float3 d;           // the watertight test keeps its own constants of d
};

// two floats in a 64-bit register pair, and the two-wide multiply-add of sm_100
typedef unsigned long long f32x2;
NB_D f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
NB_D f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
NB_D float lo2(f32x2 v) { return __uint_as_float((uint32_t)v); }
NB_D float hi2(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }

// three-operand minimum and maximum (one instruction on sm_100)
NB_D float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
NB_D float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// A wide node's visit: its entries whose box the ray may meet within tmax in
// the binary traversal's order for the ray's octant, the first into `next`,
// the rest pushed so that they come off the stack in order.  False on a stack
// overflow.
template <class Ray>
NB_D bool wide_visit(const DevNode4* nd, const uint4& meta, const Ray& r, float tmax, const SmemStack& st, int cap,
                     int& top, uint32_t& next, uint32_t* status) {
    // near and far planes picked by address (the ray's sign), two boxes at a time
    const ulonglong2* b = reinterpret_cast<const ulonglong2*>(nd->lo);
    const uint32_t sx = (r.neg & 1u) ? 3u : 0u, sy = (r.neg & 2u) ? 3u : 0u, sz = (r.neg & 4u) ? 3u : 0u;
    const ulonglong2 nx = __ldg(b + sx), fx = __ldg(b + (3u - sx));
    const ulonglong2 ny = __ldg(b + 1 + sy), fy = __ldg(b + 1 + (3u - sy));
    const ulonglong2 nz = __ldg(b + 2 + sz), fz = __ldg(b + 2 + (3u - sz));
    const uint4 child = __ldg(&nd->child);
    uint32_t w[4] = {child.x, child.y, child.z, child.w};
    const f32x2 ix = pack2(r.inv.x, r.inv.x), iy = pack2(r.inv.y, r.inv.y), iz = pack2(r.inv.z, r.inv.z);
    const f32x2 cnx = pack2(r.cn.x, r.cn.x), cny = pack2(r.cn.y, r.cn.y), cnz = pack2(r.cn.z, r.cn.z);
    const f32x2 cfx = pack2(r.cf.x, r.cf.x), cfy = pack2(r.cf.y, r.cf.y), cfz = pack2(r.cf.z, r.cf.z);
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const f32x2 tnx = fma2(h ? nx.y : nx.x, ix, cnx), tfx = fma2(h ? fx.y : fx.x, ix, cfx);
        const f32x2 tny = fma2(h ? ny.y : ny.x, iy, cny), tfy = fma2(h ? fy.y : fy.x, iy, cfy);
        const f32x2 tnz = fma2(h ? nz.y : nz.x, iz, cnz), tfz = fma2(h ? fz.y : fz.x, iz, cfz);
        const float tn0 = max3(lo2(tnx), lo2(tny), lo2(tnz)), tf0 = min3(lo2(tfx), lo2(tfy), lo2(tfz));
        const float tn1 = max3(hi2(tnx), hi2(tny), hi2(tnz)), tf1 = min3(hi2(tfx), hi2(tfy), hi2(tfz));
        if (!(tn0 <= fminf(tf0, tmax) && tf0 >= 0.0f)) w[2 * h] = kWNone;
        if (!(tn1 <= fminf(tf1, tmax) && tf1 >= 0.0f)) w[2 * h + 1] = kWNone;
    }
    // into the ray's order, nearest first
    const uint32_t f = meta.y >> (3u * (r.neg & 7u));
    const uint32_t a0 = f & 1u ? w[1] : w[0], a1 = f & 1u ? w[0] : w[1];
    const uint32_t a2 = f & 2u ? w[3] : w[2], a3 = f & 2u ? w[2] : w[3];
    const uint32_t o[4] = {f & 4u ? a2 : a0, f & 4u ? a3 : a1, f & 4u ? a0 : a2, f & 4u ? a1 : a3};
    if (top + 3 > cap) {
        // room for every entry is checked at once; near the end of the stack, for the entries there are
        int k = 0;
        for (int j = 0; j < 4; ++j) k += o[j] != kWNone;
        if (top + k - 1 > cap) {
            atomicOr(status, NOOR_DEV_STACK_OVERFLOW);
            return false;
        }
    }
    // last in order first: each taken word pushes the one held before it
    next = o[3];
#pragma unroll
    for (int j = 2; j >= 0; --j) {
        if (o[j] == kWNone) continue;
        if (next != kWNone) {
            st.base[top * st.stride] = next;
            ++top;
        }
        next = o[j];
    }
    return true;
}

// An inner node taken from the stack or a ref once its box passed: its wide
// node, or for a ray below which boxes may not be skipped one binary step
// (the far child pushed, the near one next, as trace_closest takes them).
// False on a stack overflow or a missing wide node.
NB_D bool inner_step(const DevScene& S, uint32_t ni, const uint4& lo, const uint4& hi, uint32_t neg_bits, bool deg,
                     const SmemStack& st, int cap, int& top, uint32_t& next, uint32_t* status) {
    if (deg) {
        if (top + 1 > cap) {
            atomicOr(status, NOOR_DEV_STACK_OVERFLOW);
            return false;
        }
        const bool neg = (neg_bits >> (hi.w & NOOR_AXIS_MASK)) & 1u;
        st.base[top * st.stride] = kWRef | (neg ? ni + 1 : lo.w);
        ++top;
        next = kWRef | (neg ? lo.w : ni + 1);
        return true;
    }
    next = __ldg(&S.map4[ni]);
    if (next == kWNone) {
        atomicOr(status, NOOR_DEV_BAD_INDEX);
        return false;
    }
    return true;
}

// The exact slab test of the leaf whose triangles start at `start`, made when
// one of them is hit: the leaf's box must pass with the distance the binary
// traversal would have tested it with.
template <class Ray>
NB_D bool leaf_box_hit(const DevScene& S, uint32_t start, const Ray& r, float tmax) {
    const DevNode* nd = S.nodes + __ldg(&S.leaf_of[start]);
    return slab_hit(r, __ldg(&nd->lo), __ldg(&nd->hi), tmax);
}

// The world ray of a walk, held in registers or read again from memory where
// it is needed again (an instance whose transform is not the identity, a
// light)
struct HeldRay {
    float3 o, d;
    NB_D void get(float3& oo, float3& dd) const {
        oo = o;
        dd = d;
    }
};
struct StoredRay {
    const float4 *o, *d;
    NB_D void get(float3& oo, float3& dd) const {
        const float4 a = *o, b = *d;
        oo = f3(a);
        dd = f3(b);
    }
};

// The ray of the level being walked, for the four-wide traversals.  The world
// ray is not kept beside it: it is set up again when a top-level node follows
// an instance whose transform is not the identity.
template <int ISECT>
struct LevelRay {
    BoxRay<ISECT> r;
    WtRay wt;           // watertight constants
    bool deg;           // walks the binary tree
    bool world;         // r is the world ray

    NB_D bool hit_triangle(const DevScene& S, uint32_t ti, float& t, float& bu, float& bv, uint32_t& mt) const {
        if constexpr (ISECT == NOOR_ISECT_WATERTIGHT)
            return wt_test(r, wt, S.wtri + ti, t, bu, bv, mt);
        else
            return wald_test(r, S.wald + ti, t, bu, bv, mt);
    }
    NB_D void setup(const DevScene& S, const float3& o, const float3& d, bool binary) {
        TRay t;
        tray_setup(t, o, d);
        r.o = o;
        r.inv = t.inv;
        r.neg = t.neg;
        const float e = 3.0e-7f;
        const float3 pad = f3(e * (fabsf(o.x) + S.reach4) * fabsf(t.inv.x), e * (fabsf(o.y) + S.reach4) * fabsf(t.inv.y),
                              e * (fabsf(o.z) + S.reach4) * fabsf(t.inv.z));
        r.cn = f3(fmaf(-o.x, t.inv.x, -pad.x), fmaf(-o.y, t.inv.y, -pad.y), fmaf(-o.z, t.inv.z, -pad.z));
        r.cf = f3(fmaf(-o.x, t.inv.x, pad.x), fmaf(-o.y, t.inv.y, pad.y), fmaf(-o.z, t.inv.z, pad.z));
        deg = binary || wide_degenerate(o, d);
        if constexpr (ISECT == NOOR_ISECT_WATERTIGHT)
            wt_setup(wt, d);
        else
            r.d = d;
    }
    template <class World>
    NB_D void to_world(const DevScene& S, const World& w, bool binary) {
        if (world) return;
        float3 o, d;
        w.get(o, d);
        setup(S, o, d, binary);
        world = true;
    }
    // into instance `ins`: an instance whose world-to-object rows are exactly
    // the identity (DevScene::xf_ident) leaves a plain ray as it is
    template <class World>
    NB_D void to_object(const DevScene& S, const World& w, uint32_t ins, bool binary) {
        TRay t, x;
        w.get(t.o, t.d);
        if (((__ldg(&S.xf_ident[ins >> 5]) >> (ins & 31u)) & 1u) && ray_plain(t.o, t.d)) {
            to_world(S, w, binary);
            return;
        }
        tray_to_object(x, t, S.xforms + ins);
        setup(S, x.o, x.d, binary);
        world = false;
    }
};

// Any hit over the four-wide tree (S.nodes4, layout in wide_bvh.h): the same
// answer as trace_any on the binary tree.  Refs (mesh leaves, instances,
// light nodes, deferred entries, leaves a word cannot hold) are taken as the
// binary traversal takes them.  `binary`: walk the binary tree only (a scene
// without a four-wide tree, or one whose binary stack may not fit `cap`).
// The stack holds `cap` words.
template <int ISECT, bool EXT, class World>
NB_D bool trace_any4(const DevScene& S, const World& world, float tmax, const SmemStack& st, int cap, bool binary,
                     uint32_t* status) {
    LevelRay<ISECT> L;
    {
        float3 o, d;
        world.get(o, d);
        L.setup(S, o, d, binary);
    }
    L.world = true;
    int top = 0;
    uint32_t next = L.deg ? kWRef | S.root : S.root4;
    for (;;) {
        const uint32_t cur = next;
        next = kWNone;
        if (!(cur & kWRef)) {
            const DevNode4* nd = S.nodes4 + cur;
            const uint4 meta = __ldg(&nd->meta);
            if (meta.x & kW4World) L.to_world(S, world, binary);
            if (!wide_visit(nd, meta, L.r, tmax, st, cap, top, next, status)) return false;
        } else if ((cur & (kWUntested | kWLeaf)) == kWLeaf) {
            const uint32_t start = cur & kWLeafStart, end = start + ((cur >> kWLeafShift) & (kWLeafMaxCount - 1u)) + 1u;
            for (uint32_t ti = start; ti < end; ++ti) {
                float tm = tmax, bu, bv;
                uint32_t mt;
                bool h = L.hit_triangle(S, ti, tm, bu, bv, mt);
                if (h && EXT && S.has_alpha && (mt & NOOR_ALPHA) && alpha_cut<ISECT>(S, ti, bu, bv)) h = false;
                if (h) {
                    if (leaf_box_hit(S, start, L.r, tmax)) return true;
                    break;
                }
            }
        } else if (cur & kWUntested) {
            L.to_object(S, world, cur & kWIndex, binary);
            next = __ldg(&S.inst_root[cur & kWIndex]);
        } else {
            const uint32_t ni = cur & kWIndex;
            const DevNode* nd = S.nodes + ni;
            const uint4 lo = __ldg(&nd->lo);
            const uint4 hi = __ldg(&nd->hi);
            if (hi.w & NOOR_MESH_NODE_MASK) L.to_world(S, world, binary);
            if (slab_hit(L.r, lo, hi, tmax)) {
                if (!(hi.w & kNodeKindMask)) {
                    if (!inner_step(S, ni, lo, hi, L.r.neg, L.deg, st, cap, top, next, status)) return false;
                } else if (hi.w & NOOR_LIGHT_NODE_MASK) {
                    const uint32_t li = hi.w & NOOR_LIGHT_MASK;
                    float tm = tmax;
                    float3 o, d;
                    world.get(o, d);
                    if ((int)li < S.num_area_lights &&
                        shape_hit<EXT, ISECT == NOOR_ISECT_REF_WALD>(S.area_lights[li], o, d, tm))
                        return true;
                } else if (hi.w & NOOR_MESH_INSTANCE_MASK) {
                    L.to_object(S, world, hi.w & NOOR_TRANS_MASK, binary);
                    next = kWRef | lo.w;
                } else if (hi.w & NOOR_MESH_LEAF_MASK) {
                    const uint32_t cnt = hi.w & NOOR_COUNT_MASK;
                    if (top + (int)cnt > cap + 1) {
                        atomicOr(status, NOOR_DEV_STACK_OVERFLOW);
                        return false;
                    }
                    for (uint32_t i = 1; i < cnt; ++i) {
                        st.base[top * st.stride] = kWRef | (ni + i);
                        ++top;
                    }
                    if (cnt) next = kWRef | (ni + cnt);
                } else {
                    const uint32_t start = lo.w;
                    const uint32_t end = start + (hi.w & NOOR_TRI_COUNT_MASK);
                    for (uint32_t ti = start; ti < end; ++ti) {
                        float tm = tmax, bu, bv;
                        uint32_t mt;
                        bool h = L.hit_triangle(S, ti, tm, bu, bv, mt);
                        if (h && EXT && S.has_alpha && (mt & NOOR_ALPHA) && alpha_cut<ISECT>(S, ti, bu, bv)) h = false;
                        if (h) return true;
                    }
                }
            }
        }
        if (next == kWNone) {
            if (top == 0) return false;
            --top;
            next = st.base[top * st.stride];
        }
    }
}

// Closest hit over the four-wide tree: the same hit, to the bit, as
// trace_closest.  Leaves are taken in the binary traversal's order.  A ref is
// slab-tested when it is taken and a leaf when a triangle of it is hit, both
// against the hit distance of the moment they were taken, as the binary
// traversal tests them; the widened boxes only skip what the binary
// traversal would find missed (its hit distance only shrinks, and a box
// inside a missed box is missed).
template <int ISECT, bool EXT, class World>
NB_D bool trace_closest4(const DevScene& S, const World& world, float& tmax, HitRec& rec, const SmemStack& st, int cap,
                         bool binary, uint32_t* status) {
    LevelRay<ISECT> L;
    {
        float3 o, d;
        world.get(o, d);
        L.setup(S, o, d, binary);
    }
    L.world = true;
    // the distance the level's boxes and triangles are tested with: a light
    // hit shortens tmax, and the level's follows at the next top-level node
    float ltmax = tmax;
    uint32_t ins = 0;
    bool hit = false;
    int top = 0;
    uint32_t next = L.deg ? kWRef | S.root : S.root4;
    for (;;) {
        const uint32_t cur = next;
        next = kWNone;
        if (!(cur & kWRef)) {
            const DevNode4* nd = S.nodes4 + cur;
            const uint4 meta = __ldg(&nd->meta);
            if (meta.x & kW4World) {
                L.to_world(S, world, binary);
                ltmax = tmax;
            }
            if (!wide_visit(nd, meta, L.r, ltmax, st, cap, top, next, status)) return hit;
        } else {
            uint32_t start = 0, end = 0;
            bool known = false;   // the leaf's box has passed
            if ((cur & (kWUntested | kWLeaf)) == kWLeaf) {
                start = cur & kWLeafStart;
                end = start + ((cur >> kWLeafShift) & (kWLeafMaxCount - 1u)) + 1u;
            } else if (cur & kWUntested) {
                ins = cur & kWIndex;
                L.to_object(S, world, ins, binary);
                ltmax = tmax;
                next = __ldg(&S.inst_root[ins]);
            } else {
                const uint32_t ni = cur & kWIndex;
                const DevNode* nd = S.nodes + ni;
                const uint4 lo = __ldg(&nd->lo);
                const uint4 hi = __ldg(&nd->hi);
                if (hi.w & NOOR_MESH_NODE_MASK) {
                    L.to_world(S, world, binary);
                    ltmax = tmax;
                }
                if (slab_hit(L.r, lo, hi, ltmax)) {
                    if (!(hi.w & kNodeKindMask)) {
                        if (!inner_step(S, ni, lo, hi, L.r.neg, L.deg, st, cap, top, next, status)) return hit;
                    } else if (hi.w & NOOR_LIGHT_NODE_MASK) {
                        const uint32_t li = hi.w & NOOR_LIGHT_MASK;
                        float3 o, d;
                        world.get(o, d);
                        if ((int)li < S.num_area_lights &&
                            shape_hit<EXT, ISECT == NOOR_ISECT_REF_WALD>(S.area_lights[li], o, d, tmax)) {
                            hit = true;
                            rec.ins = li;
                            rec.mtype = NOOR_MESHLIGHT | NOOR_EMITTER;
                        }
                    } else if (hi.w & NOOR_MESH_INSTANCE_MASK) {
                        ins = hi.w & NOOR_TRANS_MASK;
                        L.to_object(S, world, ins, binary);
                        ltmax = tmax;
                        next = kWRef | lo.w;
                    } else if (hi.w & NOOR_MESH_LEAF_MASK) {
                        const uint32_t cnt = hi.w & NOOR_COUNT_MASK;
                        if (top + (int)cnt > cap + 1) {
                            atomicOr(status, NOOR_DEV_STACK_OVERFLOW);
                            return hit;
                        }
                        for (uint32_t i = 1; i < cnt; ++i) {
                            st.base[top * st.stride] = kWRef | (ni + i);
                            ++top;
                        }
                        if (cnt) next = kWRef | (ni + cnt);
                    } else {
                        start = lo.w;
                        end = start + (hi.w & NOOR_TRI_COUNT_MASK);
                        known = true;
                    }
                }
            }
            const float tleaf = ltmax;
            for (uint32_t ti = start; ti < end; ++ti) {
                float tc = ltmax, bu, bv;
                uint32_t mt;
                bool h = L.hit_triangle(S, ti, tc, bu, bv, mt);
                // the hit distance is kept only past the alpha cut
                if (EXT && S.has_alpha && h && (mt & NOOR_ALPHA) && alpha_cut<ISECT>(S, ti, bu, bv)) h = false;
                if (h) {
                    if (!known && !leaf_box_hit(S, start, L.r, tleaf)) break;
                    known = true;
                    hit = true;
                    tmax = ltmax = tc;
                    rec.u = bu;
                    rec.v = bv;
                    rec.tri = ti;
                    rec.mtype = mt;
                    rec.ins = ins;
                }
            }
        }
        if (next == kWNone) {
            if (top == 0) break;
            --top;
            next = st.base[top * st.stride];
        }
    }
    return hit;
}

// Closest hit on the four-wide tree (WIDE: the kernel is launched only for
// scenes with S.closest4 set) or on the binary one
template <int ISECT, bool EXT, bool WIDE, class World>
NB_D bool trace_primary(const DevScene& S, const World& world, float& tmax, HitRec& rec, const SmemStack& st,
                        uint32_t* status) {
    if (WIDE) return trace_closest4<ISECT, EXT>(S, world, tmax, rec, st, S.stack_cap4, false, status);
    float3 o, d;
    world.get(o, d);
    return trace_closest<ISECT, EXT>(S, o, d, tmax, rec, st, status);
}

// Any hit on the four-wide tree (WIDE: launched only for scenes with
// S.nodes4 set) or on the binary one
template <int ISECT, bool EXT, bool WIDE, class World>
NB_D bool trace_shadow(const DevScene& S, const World& world, float tmax, const SmemStack& st, uint32_t* status) {
    if (WIDE) return trace_any4<ISECT, EXT>(S, world, tmax, st, S.stack_cap4, false, status);
    float3 o, d;
    world.get(o, d);
    return trace_any<ISECT, EXT>(S, o, d, tmax, st, status);
}

// Rays a warp of this launch takes at a time from a list of n: 32, or up to 4
// where the launch has warps enough for that -- the lanes of a warp walk one
// after the other where their walks part, so a short list is spread over the
// warps (150 us of extension for a few hundred scattered rays 32 to a warp, the
// last bounces of a 1920x1080 frame, take 20 one to a warp).  Beyond 4 half
// filled warps cost more issue slots than they save latency (one sample of a
// 256x256 room, 16 rays a warp: 245 us, 32: 222; of a 768x512 sky scene, 8
// spheres: 290 and 275)
NB_D uint32_t rays_per_warp(uint32_t n) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t take = max(1u, (n + warps - 1u) / warps);
    return take > 4u ? 32u : take;
}

// The walks of the adjoint's replay: the four-wide tree where the scene has one
// and the binary walk's stack fits its capacity, else the binary tree (whose stack
// overflow is reported at that capacity, and whose nodes may be of any number)
template <int ISECT, bool EXT>
NB_D bool path_closest(const DevScene& S, const float3& o, const float3& d, float& tmax, HitRec& rec,
                       const SmemStack& st, uint32_t* status) {
    if (S.frames4 == 0u) return trace_closest<ISECT, EXT>(S, o, d, tmax, rec, st, status);
    return trace_closest4<ISECT, EXT>(S, HeldRay{o, d}, tmax, rec, st, S.stack_cap4, false, status);
}
template <int ISECT, bool EXT>
NB_D bool path_any(const DevScene& S, const float3& o, const float3& d, float tmax, const SmemStack& st,
                   uint32_t* status) {
    if (S.frames4 == 0u) return trace_any<ISECT, EXT>(S, o, d, tmax, st, status);
    return trace_any4<ISECT, EXT>(S, HeldRay{o, d}, tmax, st, S.stack_cap4, false, status);
}

}  // namespace nb
