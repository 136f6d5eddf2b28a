"""The kernels a call may be rendered with (noor_route) against each other.

Frames: the megakernel's film is the one the others have to match to the bit,
through both film modes, films continued over several calls, the first-hit
point, the ray counts, and trees that are walked as binary ones (a root without
a four-wide tree, a binary stack beyond the spec's capacity).

Adjoint: the staged forward image is the replay's to the bit; the gradients
are FP32 sums of the same terms in another order, good to a few 1e-7 per step
of the sum (1e-5 of the norm over some 1e3 steps of a parameter)."""
import ctypes as C

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes
from noor_b200.adjoint import _desc, scene_parameters

from test_gpu_stages import CASES as STAGE_CASES

pytestmark = pytest.mark.gpu

WALD, WATERTIGHT = _capi.NOOR_ISECT_REF_WALD, _capi.NOOR_ISECT_WATERTIGHT
AUTO, MEGAKERNEL, STAGED = 0, 1, 2
KAHAN, LERP = 0, 1


def _sky(s):
    s.env, s.skydome_type = None, _capi.NOOR_SKY_PHYSICAL
    s.hosek = dict(turbidity=3.0, albedo=0.3, sun_lat=1.0, sun_lon=0.8, solar_scale=250.0, solar_radius_scale=2.0)
    return s


def _field(w, h, sky="map", **render):
    g, (c, r) = scenes.sphere_field(3, 12, 4)
    s = scenes.SceneData(**g, camera=dict(scenes.frame_spheres(c, r, 3, clearance=0.5), w=w, h=h),
                         render=dict(dict(spp=1, bounces=6, rr=1, mis=1), **render), skydome_type=_capi.NOOR_SKY_HDR,
                         env=scenes.env_map(3, 128, 64, peak=50.0))
    return _sky(s) if sky == "sun" else s


def _render(s, route, calls, isect, film_mode, spec):
    """film, first hits and ray counts after each of the calls (frames each)"""
    r = scenes.Renderer(s, intersector=isect, film_mode=film_mode)
    try:
        if spec:
            r.update_spec(**{k: v(r) if callable(v) else v for k, v in spec.items()})
        _capi.call("noor_route", route, 0)
        r.counters(reset=True)
        out = []
        for n in calls:
            r.path_tracer() if n == 1 else r.render(n)
            look = (C.c_float * 4)()
            _capi.call("get_lookAt", look)
            out.append((r.framebuffer().view(np.uint32), np.array(look, np.float32).view(np.uint32), r.counters(),
                        r.status()))
        return out
    finally:
        r.close()


def _other_root(r):
    """the root's first child: a tree of its own without a four-wide form"""
    return r.spec.bvh_root_node + 1


CASES = {
    "lerp_calls": (lambda: scenes.room_scene(width=67, height=35), [1, 2, 1, 3], LERP, {}),
    "lerp_textured": (lambda: scenes.textured_room_scene(width=129, height=71), [2, 1], LERP, {}),
    "kahan_continued": (lambda: _field(65, 33), [3, 1, 2], KAHAN, {}),
    "kahan_chunks": (lambda: scenes.room_scene(width=64, height=48, bounces=2), [70, 1, 33], KAHAN, {}),
    "other_root": (lambda: _field(65, 33, "sun"), [1, 2], KAHAN, dict(bvh_root_node=_other_root)),
    "other_root_textured": (lambda: scenes.textured_room_scene(width=65, height=33), [1, 2], KAHAN,
                            dict(bvh_root_node=_other_root)),
    "short_stack": (lambda: _field(65, 33), [1, 2], LERP, dict(bvh_height=1)),
}


@pytest.mark.parametrize("route", [AUTO, STAGED])
@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("name", list(CASES))
def test_films_of_every_route(name, isect, route):
    make, calls, film_mode, spec = CASES[name]
    want = _render(make(), MEGAKERNEL, calls, isect, film_mode, spec)
    got = _render(make(), route, calls, isect, film_mode, spec)
    film = want[-1][0].view(np.float32)
    assert np.isfinite(film).all() and film[..., :3].mean() > 0.005
    for k, (a, b) in enumerate(zip(want, got)):
        assert np.array_equal(a[0], b[0]), ("film", k)
        assert np.array_equal(a[1], b[1]), ("first hit", k)
        assert a[2:] == b[2:], ("rays and status", k)


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("name", list(STAGE_CASES))
def test_staged_films_of_every_size(name, isect):
    make, frames = STAGE_CASES[name]
    want = _render(make(), MEGAKERNEL, [frames], isect, KAHAN, {})
    got = _render(make(), STAGED, [frames], isect, KAHAN, {})
    assert all(np.array_equal(a, b) for a, b in zip(want[0][:2], got[0][:2]))
    assert want[0][2:] == got[0][2:]


def test_unknown_routes_are_refused():
    r = scenes.Renderer(scenes.room_scene(width=8, height=8))
    try:
        for frames, adjoint in ((-1, 0), (99, 0), (0, -1), (0, 3)):
            assert _capi.lib().noor_route(frames, adjoint) == 1
    finally:
        r.close()


def _adjoint(s, params, gi, isect, route):
    alb, rough, env = params
    h, w = s.camera["h"], s.camera["w"]
    r = scenes.Renderer(s, intersector=isect)
    try:
        _capi.call("noor_route", 0, route)
        d = _desc((w, h, s.render["spp"], 1, s.render["bounces"]), alb, rough, env)
        img = torch.zeros((h, w, 3), device="cuda")
        ga, gr = torch.zeros_like(alb), torch.zeros_like(rough)
        ge = torch.zeros_like(env) if env.numel() else None
        torch.cuda.synchronize()
        _capi.call("noor_adjoint_forward", C.byref(d), C.c_void_p(img.data_ptr()))
        _capi.call("noor_adjoint_backward", C.byref(d), C.c_void_p(gi.data_ptr()), C.c_void_p(ga.data_ptr()),
                   C.c_void_p(gr.data_ptr()), C.c_void_p(ge.data_ptr()) if ge is not None else None)
        assert r.status(reset=True) == 0
        return img, [t for t in (ga, gr, ge) if t is not None]
    finally:
        r.close()


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("what", ["materials", "field", "field_sun", "room", "no_mis"])
def test_staged_adjoint_is_the_replays(what, isect):
    if what == "materials":    # Lambert and metal, some of a triangle each
        s = scenes.adjoint_scene(seed=5, width=65, height=31, spp=5, bounces=4, count=5, level=3, env_w=64, env_h=32)
    elif what == "room":       # a quad light
        s = scenes.room_scene(width=65, height=33, mis=True)
        s.render = dict(s.render, spp=3, bounces=4, rr=4)
    else:                      # Lambert, metal and glass
        s = _field(65, 33, "sun" if what == "field_sun" else "map", spp=3, bounces=5, rr=5, mis=int(what != "no_mis"))
    params = scene_parameters(s)
    gi = torch.from_numpy(np.random.default_rng(1).normal(size=(s.camera["h"], s.camera["w"], 3)).astype(np.float32)).cuda()
    img, grads = _adjoint(s, params, gi, isect, STAGED)
    want, want_grads = _adjoint(s, params, gi, isect, MEGAKERNEL)
    assert float(want.mean()) > 0.005
    assert torch.equal(img.view(torch.int32), want.view(torch.int32))
    assert float(want_grads[0].abs().sum()) > 0
    for g, w in zip(grads, want_grads):
        assert torch.isfinite(w).all()
        assert float((g.double() - w.double()).norm()) <= 1e-5 * float(w.double().norm())
