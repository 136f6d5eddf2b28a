"""Workloads of the render path, as a user's program calls it: listed() and
draw() describe them, prepare() makes what the program has in hand before
the call, run() is one pass through the public entry points, work() what a
pass cannot do without and exact() the 64-bit values of a pass where plain
torch gives them.

Four kinds of program use the library:
  viewer   an interactive window: load_cuda_data once, then per refresh
           cuda_path_tracer (or noor_render_frames for a burst of samples) and
           the film, with the camera or the sun moved before it
  offline  finished frames through the batched wavefront integrator
  adjoint  an optimisation step through the differentiable renderer
  rays     ray queries (picking, visibility) and payload builds of scene tools
"""
import ctypes as C
import math

import numpy as np
import torch

from noor_b200 import _capi as capi
from noor_b200 import adjoint, scenes


# ------------------------------------------------------------------ cases
def _viewer(name, scene, width, height, frames, **kw):
    d = dict(name=name, kind="viewer", scene=scene, width=width, height=height, frames=frames, bounces=8, count=32,
             level=6, mis=False, isect=0, film=0, move="camera")
    d.update(kw)
    return d


def _offline(name, scene, width, height, spp, **kw):
    d = dict(name=name, kind="offline", scene=scene, width=width, height=height, spp=spp, bounces=8, count=32,
             level=6, mis=False, slots=1 << 24, block=64, sort=2)
    d.update(kw)
    return d


def listed():
    return [
        # the window of a small scene while its camera is dragged: one sample
        # per pixel per refresh, the call's latency is what the user feels
        _viewer("viewer_room", "room", 256, 256, 1, bounces=5),
        # the same window over a large scene at full size
        _viewer("viewer_sky", "sky", 1920, 1080, 1),
        # the sun dragged: a new sky fitted, its distribution rebuilt, a frame
        _viewer("viewer_sun", "sky", 960, 540, 1, count=8, level=5, mis=True, move="sun"),
        # textures, bump and alpha maps, the reference's own triangle test and
        # running-mean film, an odd window size, a burst of samples
        _viewer("viewer_textured", "textured", 641, 359, 4, bounces=5, isect=1, film=1),
        # a still converging under an environment map with MIS
        _viewer("still_env", "env", 960, 540, 16, count=16, level=5, mis=True),
        # offline frames: the smallest configuration, the headline one, the
        # environment-lit one
        _offline("offline_room", "room", 256, 256, 16, bounces=5, slots=1 << 20, sort=1),
        _offline("offline_sky", "sky", 1920, 1080, 64),
        _offline("offline_env", "env", 1920, 1080, 32, mis=True),
        # many uneven frames of several scenes in one launch
        dict(name="offline_batch", kind="batch", frames=12, side_min=128, side_max=1024, spp_max=48, bounces=6,
             count=12, level=5, slots=1 << 22, block=64, sort=2),
        # one optimisation step: render, loss, gradients of materials and map
        dict(name="adjoint_step", kind="adjoint", width=512, height=512, spp=16, bounces=4, count=10, level=5,
             materials=64, env_w=512, env_h=256),
        # scattered ray queries on a large scene, closest hit and visibility
        dict(name="ray_queries", kind="rays", scene="sky", n=1 << 20, count=32, level=6, isect=0),
        # a scene tool's payload build on the device
        dict(name="payload_build", kind="build", count=16, level=6),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["viewer", "viewer", "offline", "offline", "batch", "adjoint", "rays", "build"])
    level = rng.randint(3, 6)
    count = log_int(2, 32)
    if kind == "viewer":
        scene = rng.choice(["room", "sky", "env", "textured"])
        d = _viewer("", scene, log_int(97, 1920), log_int(61, 1080), log_int(1, 8), count=count, level=level,
                    bounces=rng.randint(2, 8), mis=scene == "env" or rng.random() < 0.3, isect=int(rng.random() < 0.3),
                    film=int(rng.random() < 0.3), move="sun" if scene == "sky" and rng.random() < 0.3 else "camera")
    elif kind == "offline":
        scene = rng.choice(["room", "sky", "env"])
        d = _offline("", scene, log_int(97, 1920), log_int(61, 1080), log_int(3, 48), count=count, level=level,
                     bounces=rng.randint(2, 8), mis=scene == "env", slots=1 << rng.randint(18, 22),
                     block=rng.choice([32, 64, 128]), sort=rng.randint(0, 3))
    elif kind == "batch":
        d = dict(kind="batch", frames=rng.randint(2, 12), side_min=64, side_max=log_int(128, 768),
                 spp_max=log_int(4, 32), bounces=rng.randint(2, 6), count=rng.randint(2, 8), level=rng.randint(3, 5),
                 slots=1 << rng.randint(18, 22), block=rng.choice([32, 64, 128]), sort=rng.randint(0, 3))
    elif kind == "adjoint":
        d = dict(kind="adjoint", width=log_int(33, 400), height=log_int(33, 400), spp=log_int(1, 16),
                 bounces=rng.randint(1, 4), count=rng.randint(3, 10), level=rng.randint(3, 5),
                 materials=rng.randint(2, 64), env_w=log_int(16, 512), env_h=log_int(8, 256))
    elif kind == "rays":
        d = dict(kind="rays", scene=rng.choice(["room", "sky"]), n=log_int(1000, 1 << 20), count=count, level=level,
                 isect=int(rng.random() < 0.5))
    else:
        d = dict(kind="build", count=log_int(1, 16), level=rng.randint(2, 6))
    d.pop("name", None)
    return d


# ---------------------------------------------------------------- prepare
class Session:
    """One render context of the library (scene, sky, camera, spec) and what
    the program keeps alive for it; bind() makes it the thread's current one."""

    def __init__(self, scene, isect=0, film=0):
        self.scene = scene
        self.context = None
        built = scenes.BuiltPayload(scene, gpu=True)
        self.spec = built.default_spec(scene.render["bounces"], scene.render["rr"])
        self.spec.mis = int(scene.render["mis"])
        self.spec.intersector, self.spec.film_mode = isect, film
        self.camera = scenes.make_camera(scene.camera)
        self.hosek = scenes.make_hosek(scene.hosek)
        self.built = built
        capi.call("noor_context_bind", None)
        capi.call("load_cuda_data", C.byref(built.payload), C.byref(self.hosek), C.byref(self.camera),
                  C.byref(self.spec), None)
        self.context = capi.lib().noor_context_current()

    def bind(self):
        capi.call("noor_context_bind", self.context)

    def __del__(self):
        if self.context:
            now = capi.lib().noor_context_current()
            capi.lib().noor_context_bind(self.context)
            capi.lib().device_free_memory()
            capi.lib().noor_context_bind(None if now == self.context else now)
            self.context = None


def _sky(rng):
    """sun position and turbidity of a seeded day"""
    return dict(turbidity=float(rng.uniform(2.0, 5.0)), albedo=0.3, sun_lat=float(np.radians(rng.uniform(30.0, 70.0))),
                sun_lon=float(rng.uniform(0.0, 2 * np.pi)), solar_scale=250.0, solar_radius_scale=2.0)


def _scene(case, seed, width, height, spp):
    """the SceneData of a case: generators of noor_b200.scenes, seeded"""
    kw = dict(width=width, height=height, spp=spp, bounces=case["bounces"])
    if case["scene"] == "room":
        return scenes.room_scene(seed=seed, **kw)
    if case["scene"] == "textured":
        return scenes.textured_room_scene(seed=seed, **kw)
    g, (c, r) = scenes.sphere_field(seed, case["count"], case["level"])
    if case["count"] == 1:
        cam = dict(eye=tuple(c[0] + r[0] * np.array([0.0, 1.0, 3.0])), look_at=tuple(c[0]), up=(0.0, 1.0, 0.0),
                   fov_deg=50.0, w=width, h=height)
    else:
        cam = dict(scenes.frame_spheres(c, r, seed, clearance=0.5), w=width, h=height)
    render = dict(spp=spp, bounces=case["bounces"], rr=1, mis=int(case["mis"]))
    if case["scene"] == "env":
        return scenes.SceneData(**g, skydome_type=capi.NOOR_SKY_HDR, env=scenes.env_map(seed, 1024, 512, peak=100.0),
                                camera=cam, render=render, name="env")
    return scenes.SceneData(**g, skydome_type=capi.NOOR_SKY_PHYSICAL, camera=cam, render=render,
                            hosek=_sky(np.random.default_rng(seed)), name="sky")


def _film(height, width):
    return torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")


def _batch_sizes(case):
    """(width, height, spp) of a batch's frames: the job's own, whatever its scenes"""
    rng = np.random.default_rng(case["frames"] * 10007 + case["side_max"])
    out = []
    for _ in range(case["frames"]):
        w = int(round(math.exp(rng.uniform(math.log(case["side_min"]), math.log(case["side_max"])))))
        out.append((w, max(case["side_min"], int(w * rng.uniform(0.5, 1.0))), int(rng.integers(4, case["spp_max"] + 1))))
    return out


def prepare(case, seed):
    state = dict(case=case)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "viewer":
        s = state["session"] = Session(_scene(case, seed, case["width"], case["height"], case["frames"]),
                                       case["isect"], case["film"])
        state["film"] = _film(case["height"], case["width"])
        state["table"] = np.ascontiguousarray(scenes.hosek_dataset())
        state["suns"] = [_sky(rng) for _ in range(2)]
        state["passes"] = 0
        assert s.context
    elif kind == "offline":
        state["session"] = Session(_scene(case, seed, case["width"], case["height"], case["spp"]))
        film = state["film"] = _film(case["height"], case["width"])
        state["frames"] = (capi.WfFrame * 1)(scenes.wf_frame(0, state["session"].scene.camera, case["spp"],
                                                             case["bounces"], d_film=film.data_ptr()))
        state["params"] = scenes.wf_params(case["block"], case["slots"], case["sort"], 1)
    elif kind == "batch":
        # two fields and two single objects, under a sky or an environment map
        small = dict(case, count=1, scene="sky", mis=False)
        made = [_scene(dict(case, scene="sky", mis=False), seed, 64, 64, 1), _scene(small, seed + 1, 64, 64, 1),
                _scene(dict(case, scene="env", mis=True), seed + 2, 64, 64, 1),
                _scene(dict(small, scene="env", mis=True), seed + 3, 64, 64, 1)]
        s = state["session"] = Session(made[0])
        ids, state["keep"] = [0], []
        for sd in made[1:]:
            i, keep = scenes.upload_scene(sd, built=scenes.BuiltPayload(sd, gpu=True))
            ids.append(i)
            state["keep"].append(keep)
        frames, films = [], []
        for w, h, spp in _batch_sizes(case):
            k = int(rng.integers(0, len(made)))
            films.append(_film(h, w))
            frames.append(scenes.wf_frame(ids[k], dict(made[k].camera, w=w, h=h), spp, case["bounces"],
                                          d_film=films[-1].data_ptr()))
        state["film"], state["frames"] = films, (capi.WfFrame * len(frames))(*frames)
        state["params"] = scenes.wf_params(case["block"], case["slots"], case["sort"], 1)
    elif kind == "adjoint":
        sd = scenes.adjoint_scene(seed, case["width"], case["height"], case["spp"], case["bounces"], case["count"],
                                  case["level"], case["materials"], case["env_w"], case["env_h"])
        state["session"] = Session(sd)
        state["params"] = [t.requires_grad_(True) for t in adjoint.scene_parameters(sd)]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # the picture the step pulls towards
        state["target"] = torch.rand((case["height"], case["width"], 3), device="cuda", generator=g)
    elif kind == "rays":
        state["session"] = Session(_scene(dict(case, bounces=4, mis=False), seed, 64, 64, 1), case["isect"])
        rays = torch.from_numpy(_rays(case, seed)).cuda()
        state["rays"], n = rays, case["n"]
        state["short"] = rays.clone()
        state["short"][:, 3] = 4.0   # visibility within a few units
        state["hits"] = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
        state["blocked"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    else:
        g, _ = scenes.sphere_field(seed, case["count"], case["level"])
        sd = scenes.SceneData(**g)
        state["desc"], state["keep"] = scenes.scene_desc(sd)
        n = sd.num_triangles
        state["order"] = np.zeros(n, np.uint32)
        state["lo"], state["hi"] = (np.zeros((2 * n + 4 * case["count"] + 16, 4), np.int32) for _ in range(2))
    torch.cuda.synchronize()
    return state


def _rays(case, seed):
    """(n, 8) noor_ray records: origins through the scene's volume, every direction"""
    rng = np.random.default_rng(seed + 7)
    n = case["n"]
    lo, hi = ((-0.95, 0.05, -0.95), (0.95, 1.95, 0.95)) if case["scene"] == "room" else ((-10.0,) * 3, (10.0,) * 3)
    r = np.zeros((n, 8), np.float32)
    r[:, :3] = rng.uniform(lo, hi, (n, 3))
    r[:, 3] = np.inf
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return r


# -------------------------------------------------------------------- run
def _ptr(t):
    return C.c_void_p(t.data_ptr())


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "build":
        return _build(state)
    s = state["session"]
    s.bind()
    if kind == "viewer":
        frame = C.c_uint(1)
        if case["move"] == "sun":
            h = state["suns"][state["passes"] % 2]
            albedo = (C.c_float * 3)(h["albedo"], h["albedo"], h["albedo"])
            capi.call("noor_hosek_fit", state["table"].ctypes.data_as(capi.pf), h["turbidity"], albedo, h["sun_lat"],
                      h["sun_lon"], h["solar_scale"], h["solar_radius_scale"], C.byref(s.hosek))
            capi.call("update_cuda_hosek")
        else:
            capi.call("update_cuda_camera")
        state["passes"] += 1
        if case["frames"] == 1:
            capi.call("cuda_path_tracer", C.byref(frame))
        else:
            capi.call("noor_render_frames", C.byref(frame), case["frames"])
        capi.call("noor_get_framebuffer_device", _ptr(state["film"]), case["width"] * case["height"])
        return state["film"]
    if kind in ("offline", "batch"):
        capi.call("noor_wavefront_render", state["frames"], len(state["frames"]), C.byref(state["params"]))
        return state["film"]
    if kind == "adjoint":
        params = state["params"]
        for p in params:
            p.grad = None
        img = adjoint.render(*params, case["width"], case["height"], case["spp"])
        ((img - state["target"]) ** 2).sum().backward()
        return dict(image=img.detach(), albedo=params[0].grad, roughness=params[1].grad, env=params[2].grad)
    capi.call("noor_trace_closest", _ptr(state["rays"]), _ptr(state["hits"]), case["n"])
    capi.call("noor_trace_any", _ptr(state["short"]), _ptr(state["blocked"]), case["n"])
    hits = state["hits"]
    hit = hits[:, 6]
    words = torch.where(hit[:, None] != 0, hits, torch.zeros_like(hits))   # a miss leaves t at the ray's extent
    return dict(index=words[:, 1:4], hit=hit, t=words[:, 0].contiguous().view(torch.float32),
                uv=words[:, 4:6].contiguous().view(torch.float32), blocked=state["blocked"])


class _Payload:
    """a built payload and the host arrays the library owns for it"""

    def __init__(self, desc):
        self.handle, self.view, stat = C.c_void_p(), capi.Payload(), capi.BuildStat()
        capi.call("noor_build_payload_gpu", C.byref(desc), C.byref(self.handle), C.byref(stat))
        capi.call("noor_payload_view", self.handle, C.byref(self.view))

    def __del__(self):
        if self.handle.value:
            capi.lib().noor_free_payload(self.handle)

    def words(self, pointer, rows):
        """(rows, 4) words of a library array, read in place (floats as their bits)"""
        block = (C.c_int32 * (4 * rows)).from_address(C.cast(pointer, C.c_void_p).value)
        block.payload = self   # the array lives as long as what reads it
        return np.frombuffer(block, np.int32).reshape(rows, 4)


def _build(state):
    p = _Payload(state["desc"])
    v, n, nodes = p.view, p.view.num_triangles, p.view.num_bvh_nodes
    capi.call("noor_payload_triangle_order", p.handle, state["order"].ctypes.data_as(capi.pu), n)
    # the node arrays into the tool's own, sized for any tree over these triangles
    lo, hi = state["lo"], state["hi"]
    lo[:nodes] = p.words(v.bvh_min_right_start, nodes)
    hi[:nodes] = p.words(v.bvh_max_axis_count, nodes)
    return dict(order=state["order"].view(np.int32), nodes=nodes, lo=lo, hi=hi,
                attributes=p.words(v.attribute_indices, n), wald=p.words(v.wald_ax_nu_nv_nd, n),
                wald_b=p.words(v.wald_bnu_bnv_au_av, n), wald_c=p.words(v.wald_cnu_cnv_deg_mat, n),
                vertices=p.words(v.vertices, v.num_vertices), normals=p.words(v.normals, v.num_vertices))


# ------------------------------------------------------------------- work
def _triangles(case):
    if case.get("scene") in ("room", "textured"):
        return 38
    return case["count"] * 20 * 4 ** case["level"]


def work(case):
    """What a pass cannot do without: every input read once and every output
    written once; per ray a path down a binary tree (slab tests of both
    children per level, 30 operations) and two triangle tests (50 each), per
    surface hit some 300 operations of shading.  A path has about two and a
    half extension rays and, where lights are sampled, one shadow ray each."""
    kind, tris = case["kind"], _triangles(case)
    scene = tris * (48 + 32 + 16) + 3 * tris * 8
    walk = 30.0 * math.log2(tris) + 100.0
    if kind == "build":
        # triangle boxes and centroids binned at every level of the tree; triples of indices and
        # vertices in, nodes, records and de-duplicated vertices out
        return dict(bytes=tris * (36 + 4 + 0.5 * 32) + tris * (16 * 4 + 4 + 0.5 * 32 + 32),
                    flops=tris * math.log2(max(tris, 2)) * 12.0)
    if kind == "rays":
        return dict(bytes=scene + case["n"] * (32 + 32 + 32 + 4), flops=2 * case["n"] * walk)
    if kind == "batch":
        sizes = _batch_sizes(case)
        paths, film = sum(w * h * spp for w, h, spp in sizes), sum(w * h for w, h, _ in sizes) * 16
        scene *= 2.2
    else:
        px = case["width"] * case["height"]
        paths, film = px * case.get("spp", case.get("frames", 1)), px * 16
    rays = min(2.5, case["bounces"]) * (2 if case.get("mis") or case.get("scene") in ("room", "textured") else 1.5)
    flops = paths * rays * (walk + 300.0)
    if kind == "adjoint":
        # rendered once and replayed once more for the gradients; image out, its gradient in
        env = case["env_w"] * case["env_h"] * 12
        return dict(bytes=scene + px * 24 + 2 * env, flops=2 * flops)
    if case.get("move") == "sun":
        flops += 2048 * 1024 * 16 * 60.0   # the sky's cells, 4 x 4 samples each
    return dict(bytes=scene + film, flops=flops)


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """Ray queries against every triangle in 64 bits (a ray is tested against
    the triangles of the objects whose bounding sphere it meets).  Renders and
    gradients are sums over seeded random paths, which have no value outside
    the renderer; payloads are whole numbers."""
    if case["kind"] != "rays":
        return None
    s = _scene(dict(case, bounces=4, mis=False), seed, 64, 64, 1)
    groups = [(0, s.num_triangles)] if case["scene"] == "room" else [(m["tri_start"], m["tri_count"]) for m in s.meshes]
    f64 = dict(dtype=torch.float64, device="cuda")
    V = torch.tensor(s.vertices[:, :3], **f64)
    tri = torch.from_numpy(s.vindices.astype(np.int64)).cuda()
    rays = torch.from_numpy(_rays(case, seed)).cuda().double()
    o, d = rays[:, :3], rays[:, 4:7]
    best = torch.full((case["n"],), math.inf, **f64)
    for start, count in groups:
        P = V[tri[start:start + count]]                        # (m, 3, 3)
        mid = P.reshape(-1, 3).mean(0)
        rad = (P.reshape(-1, 3) - mid).norm(dim=1).max() * (1 + 1e-6)
        along = ((mid - o) * d).sum(1).clamp(min=0)
        near = ((o + along[:, None] * d - mid).norm(dim=1) <= rad).nonzero()[:, 0]
        a, e1, e2 = P[:, 0], P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
        n = torch.linalg.cross(e1, e2)
        # per triangle six row vectors against the ray's (d, o x d): determinant and barycentrics as products
        Q = torch.cat([torch.linalg.cross(a, e2), e2, -torch.linalg.cross(a, e1), -e1], 1)
        an = (a * n).sum(1)
        step = max(1, (1 << 25) // count)
        for at in range(0, near.numel(), step):
            r = near[at:at + step]
            od, dd = o[r], d[r]
            m = torch.linalg.cross(od, dd)
            det = -(dd @ n.T)
            u = dd @ Q[:, :3].T + m @ Q[:, 3:6].T
            v = dd @ Q[:, 6:9].T + m @ Q[:, 9:12].T
            t = (od @ n.T - an) / det
            u, v = u / det, v / det
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
            best[r] = torch.minimum(best[r], torch.where(ok, t, torch.full_like(t, math.inf)).min(1).values)
    t = torch.where(torch.isinf(best), torch.zeros_like(best), best)
    return dict(index=None, hit=None, t=t, uv=None, blocked=None)
