"""Bounce limits beyond what the paths of a frame make: the staged renderer
asks every 8 bounces what is left and ends with the last path.  The film, the
first hits and the ray counts are the megakernel's, with limits on and off the
asking and with paths left or not, for every kernel of the dispatch and for
trees walked as binary ones; the launches do not grow with the limit."""
import ctypes as C

import numpy as np
import pytest

from noor_b200 import _capi, scenes

from test_gpu_routes import KAHAN, LERP, MEGAKERNEL, STAGED, WALD, WATERTIGHT, _field, _other_root, _render, _sky

pytestmark = pytest.mark.gpu


def _glass(w, h, bounces):
    """paths that stay inside glass, roulette late"""
    g, (c, r) = scenes.sphere_field(5, 6, 4, kinds=("glass",), box=4.0, rmin=0.8)
    return _sky(scenes.SceneData(**g, camera=dict(scenes.frame_spheres(c, r, 3, clearance=0.5), w=w, h=h),
                                 render=dict(spp=1, bounces=bounces, rr=12, mis=1)))


def _bright_room(w, h, bounces):
    """every path goes on until the roulette of bounce 30"""
    s = scenes.room_scene(width=w, height=h, bounces=bounces)
    s.render = dict(s.render, rr=30)
    return s


CASES = {
    "room": (lambda b: scenes.room_scene(width=97, height=61, bounces=b), [2], KAHAN, {}),
    "many_left": (lambda b: _bright_room(600, 401, b), [1, 1], LERP, {}),
    "glass": (lambda b: _glass(129, 97, b), [1, 2], KAHAN, {}),
    "field_mis": (lambda b: _field(161, 90, "sun", bounces=b), [3], KAHAN, {}),
    "textured": (lambda b: scenes.textured_room_scene(width=129, height=71, bounces=b), [1, 3], KAHAN, {}),
    "light": (lambda b: scenes.room_scene(width=65, height=33, light="sphere", mis=True, bounces=b), [3], KAHAN, {}),
    "binary": (lambda b: _field(65, 33, "sun", bounces=b), [2], KAHAN, dict(bvh_root_node=_other_root)),
}


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("bounces", [8, 9, 16, 17, 200])
@pytest.mark.parametrize("name", list(CASES))
def test_film_at_a_bounce_limit(name, bounces, isect):
    make, calls, film, spec = CASES[name]
    want = _render(make(bounces), MEGAKERNEL, calls, isect, film, spec)
    got = _render(make(bounces), STAGED, calls, isect, film, spec)
    assert np.isfinite(want[-1][0].view(np.float32)).all()
    for a, b in zip(want, got):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("make", [lambda b: scenes.room_scene(width=640, height=480, bounces=b),
                                  lambda b: _field(900, 600, "sun", bounces=b)])
def test_launches_do_not_grow_with_the_limit(make):
    n = []
    for bounces in (40, 1024):
        r = scenes.Renderer(make(bounces))
        try:
            _capi.call("noor_route", STAGED, 0)
            counts = [C.c_uint64(), C.c_uint64()]
            _capi.call("noor_launch_count", C.byref(counts[0]))
            r.path_tracer()
            _capi.call("noor_launch_count", C.byref(counts[1]))
            n.append(counts[1].value - counts[0].value)
        finally:
            r.close()
    assert n[1] <= n[0] <= 5 + 2 * 40


def test_adjoint_launches_do_not_grow_with_the_limit():
    import torch
    from noor_b200.adjoint import _desc, scene_parameters
    w, h, spp = 33, 17, 2
    s = scenes.adjoint_scene(seed=5, width=w, height=h, spp=spp, bounces=1024, count=5, level=3, env_w=64, env_h=32)
    r = scenes.Renderer(s)
    alb, rough, env = scene_parameters(s)
    gi = torch.ones((h, w, 3), device="cuda")
    n, images, grads = [], [], []
    try:
        for bounces in (48, 1024):
            d = _desc((w, h, spp, 1, bounces), alb, rough, env)
            img = torch.zeros((h, w, 3), device="cuda")
            g = [torch.zeros_like(t) for t in (alb, rough, env)]
            torch.cuda.synchronize()
            at = [C.c_uint64(), C.c_uint64()]
            _capi.call("noor_launch_count", C.byref(at[0]))
            _capi.call("noor_adjoint_forward", C.byref(d), C.c_void_p(img.data_ptr()))
            _capi.call("noor_adjoint_backward", C.byref(d), C.c_void_p(gi.data_ptr()),
                       *[C.c_void_p(t.data_ptr()) for t in g])
            _capi.call("noor_launch_count", C.byref(at[1]))
            n.append(at[1].value - at[0].value)
            images.append(img)
            grads.append(g)
        assert n[1] == n[0] < 2 * (4 + 2 * 48)
        assert torch.equal(images[0], images[1])
        for x, y in zip(*grads):
            assert float((x - y).norm()) <= 1e-5 * float(x.norm())
    finally:
        r.close()
