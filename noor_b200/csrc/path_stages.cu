// Host side of the staged renderer: buffers, batches of frames, the film fold
#include <algorithm>

#include "host_common.h"
#include "path_stages.cuh"
#include "runtime.h"

namespace nb {

cudaError_t launch_stages_wt(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count, uint64_t* launches,
                             cudaStream_t s);
cudaError_t launch_stages_wald(const DevScene& S, const DevCamera& C, const StageDev& W, int sm_count,
                               uint64_t* launches, cudaStream_t s);

NB_D void stage_kahan(float3& sum, float3& c, const float3& x) {
    const float3 y = x - c;
    const float3 t = sum + y;
    c = (t - sum) - y;
    sum = t;
}

// A pixel's samples of the batch into the film, as the megakernel and
// fold_partials add them: Kahan sums over each chunk of frames in frame order,
// the chunks folded in order (one chunk: straight into the film), or the
// running mean.  The chunk in progress at the end of a batch is kept in
// part_sum / part_comp.
__global__ void __launch_bounds__(256) st_fold(DevCamera C, StageDev W, StageFold F) {
    stage_follow();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) {
        // ray counts of the batch (extend traced every active path of a bounce)
        unsigned long long ext = W.paths, sh = 0;
        for (uint32_t b = 0; b < F.bounces; ++b) {
            if (b) ext += W.count[b * kStWords + kStActive];
            sh += W.count[b * kStWords + kStShadow];
        }
        W.counters[0] += ext;
        W.counters[1] += sh;
        W.counters[2] += W.paths;
    }
    if (q >= C.w * C.h) return;
    const uint32_t pix = stage_pixel(q, C.w, C.h);
    const uint32_t per = (F.total + F.chunks - 1) / F.chunks;
    const bool blank = F.first == 0 && F.fresh;
    float3 fs = f3(0.0f), fc = f3(0.0f), sum = f3(0.0f), comp = f3(0.0f);
    float4 mean = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    if (!blank) {
        const float4 s = F.film_sum[pix];
        fs = f3(s);
        mean = s;
        if (F.film_mode == NOOR_FILM_KAHAN) fc = f3(F.film_comp[pix]);
    }
    if (F.chunks > 1u && F.first % per != 0u) {
        sum = f3(F.part_sum[pix]);
        comp = f3(F.part_comp[pix]);
    }
    for (uint32_t k = 0; k < W.frames; ++k) {
        const float3 L = f3(W.L[(size_t)q * W.frames + k]);
        const uint32_t f = F.first + k;
        if (F.film_mode != NOOR_FILM_KAHAN) {
            const uint32_t frame = F.frame0 + f;
            const float4 old = frame > 1u ? mean : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            const float t = 1.0f / (float)frame;
            mean = make_float4(old.x + t * (L.x - old.x), old.y + t * (L.y - old.y), old.z + t * (L.z - old.z),
                               old.w + t * (1.0f - old.w));
        } else if (F.chunks == 1u) {
            stage_kahan(fs, fc, L);
        } else {
            stage_kahan(sum, comp, L);
            if ((f + 1u) % per == 0u || f + 1u == F.total) {
                stage_kahan(fs, fc, sum);
                stage_kahan(fs, fc, -1.0f * comp);
                sum = comp = f3(0.0f);
                // chunks beyond the last frame fold zeros
                for (uint32_t c = f / per + 1u; f + 1u == F.total && c < F.chunks; ++c) {
                    stage_kahan(fs, fc, sum);
                    stage_kahan(fs, fc, -1.0f * comp);
                }
            }
        }
    }
    if (F.film_mode != NOOR_FILM_KAHAN) {
        F.film_sum[pix] = mean;
    } else {
        F.film_sum[pix] = make_float4(fs.x, fs.y, fs.z, 1.0f);
        F.film_comp[pix] = make_float4(fc.x, fc.y, fc.z, 0.0f);
        if (F.chunks > 1u) {
            F.part_sum[pix] = make_float4(sum.x, sum.y, sum.z, 0.0f);
            F.part_comp[pix] = make_float4(comp.x, comp.y, comp.z, 0.0f);
        }
    }
    if (pix == C.center) {
        // the last chunk's last first hit, marked by whether the last frame hit
        const uint32_t fb = (F.chunks - 1u) * per;
        float4 look = F.first > fb ? *F.lookat : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t k = 0; k < W.frames; ++k) {
            if (F.first + k < fb) continue;
            const float4 h = W.first[k];
            if (h.w != 0.0f) look = h;
            look.w = h.w;
        }
        *F.lookat = look;
    }
}

// paths a batch holds at most: 228 bytes of state each (64 more with bump
// maps), a gigabyte in all; a frame beyond it is left to the megakernel
constexpr uint32_t kStageMaxPaths = 1u << 22;

// The buffers of batches of `frames` frames, or of the most frames below that
// (halved at each try) that the device has room for and the context's limit
// allows, laid out in one allocation that the context keeps; stream-ordered, so
// that a larger one takes over what is given back for it (a first 256x256 frame
// 0.62 ms with cudaMalloc, 0.29 from a pool that holds memory).  Returns the
// frames; 0 where there is no room for one.
static uint32_t stage_buffers(Context& C, uint32_t npix, uint32_t frames, uint32_t bounces, bool diff, StageDev& W) {
    size_t at, o, d, beta, L, pend, pbeta, hit, hit2, q0, q1, qshade, qshadow, sho, shd, df, cnt, first;
    auto place = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) & ~(size_t)255;
        return p;
    };
    for (;; frames /= 2) {
        if (frames == 0) return 0;
        const size_t n = (size_t)npix * frames;
        at = 0;
        o = place(16 * n), d = place(16 * n), beta = place(16 * n), L = place(16 * n), pend = place(32 * n);
        pbeta = place(16 * n), hit = place(16 * n), hit2 = place(8 * n), q0 = place(4 * n), q1 = place(4 * n);
        qshade = place(4 * n * kStageKinds), qshadow = place(8 * n), sho = place(32 * n), shd = place(32 * n);
        df = place(diff ? 64 * n : 0), cnt = place(4 * (size_t)kStWords * (bounces + 1));
        first = place(16 * (size_t)frames);
        if (at <= C.stage_bytes) break;
        if (at > C.workspace_limit) continue;
        if (C.stage_buf) cudaFreeAsync(C.stage_buf, C.stream);
        C.stage_bytes = 0;
        if (cudaMallocAsync(&C.stage_buf, at, C.stream) == cudaSuccess) {
            C.stage_bytes = at;
            break;
        }
        cudaGetLastError();
        C.stage_buf = nullptr;
    }
    char* p = static_cast<char*>(C.stage_buf);
    W.o = (float4*)(p + o);
    W.d = (float4*)(p + d);
    W.beta = (float4*)(p + beta);
    W.L = (float4*)(p + L);
    W.pend = (float4*)(p + pend);
    W.pbeta = (float4*)(p + pbeta);
    W.hit = (float4*)(p + hit);
    W.hit2 = (uint2*)(p + hit2);
    W.diff = diff ? (float4*)(p + df) : nullptr;
    W.queue[0] = (uint32_t*)(p + q0);
    W.queue[1] = (uint32_t*)(p + q1);
    W.qshade = (uint32_t*)(p + qshade);
    W.qshadow = (uint32_t*)(p + qshadow);
    W.sh_o = (float4*)(p + sho);
    W.sh_d = (float4*)(p + shd);
    W.count = (uint32_t*)(p + cnt);
    W.first = (float4*)(p + first);
    W.cap = npix * frames;
    return frames;
}

// Frames a.frame0 .. + a.nframes - 1 into the film, staged.  *done = false
// (and nothing launched) where the megakernel has to render them.
int render_staged(Context& C, const DevScene& S, const MegaArgs& a, bool* done) {
    *done = false;
    const uint64_t npix = (uint64_t)C.cam.w * C.cam.h;
    if (npix > kStageMaxPaths || S.bounces == 0 || S.bounces > 1024) return NOOR_OK;
    if (!S.frames4 && !ref_words_fit(S.num_nodes)) return NOOR_OK;
    StageDev W{};
    const uint32_t nb = stage_buffers(C, (uint32_t)npix, (uint32_t)std::min<uint64_t>(a.nframes, kStageMaxPaths / npix),
                                      S.bounces, S.has_bump != 0u, W);
    if (nb == 0) return NOOR_OK;
    W.status = C.status;
    W.counters = C.counters;
    for (uint32_t f = 0; f < a.nframes; f += nb) {
        W.frames = std::min(nb, a.nframes - f);
        W.paths = (uint32_t)npix * W.frames;
        W.frame0 = a.frame0 + f;
        // the counters and the first hits lie side by side
        W.zero = (uint32_t)(((char*)(W.first + W.frames) - (char*)W.count) / 4);
        cudaError_t e = S.isect == NOOR_ISECT_WATERTIGHT
                            ? launch_stages_wt(S, C.cam, W, C.sm_count, &C.launches, C.stream)
                            : launch_stages_wald(S, C.cam, W, C.sm_count, &C.launches, C.stream);
        if (e != cudaSuccess) return cuda_fail(e, "staged render");
        StageFold F{};
        F.first = f;
        F.total = a.nframes;
        F.chunks = a.chunks;
        F.frame0 = a.frame0;
        F.fresh = a.fresh;
        F.film_mode = (int)S.film_mode;
        F.film_sum = a.film_sum;
        F.film_comp = a.film_comp;
        F.part_sum = a.part_sum;
        F.part_comp = a.part_comp;
        F.lookat = a.lookat;
        F.bounces = S.bounces;
        e = launch_stage(st_fold, dim3((uint32_t)((npix + 255) / 256)), 256, 0, C.stream, C.cam, W, F);
        if (e != cudaSuccess) return cuda_fail(e, "staged render");
        C.launches += 1;
    }
    *done = true;
    return NOOR_OK;
}

}  // namespace nb
