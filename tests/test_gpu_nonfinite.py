"""Throughputs that leave FP32's range.  A vertex adds throughput times direct
light to a path's radiance also where no light reaches it, so an infinite
throughput turns the radiance into NaN and the sample into 0: in every kernel
of the frames and of the adjoint alike, to the bit.  Albedos of 1e20 overflow
after a bounce or two; the other materials of the scene stay ordinary."""
import ctypes as C

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes

from test_gpu_routes import KAHAN, LERP, MEGAKERNEL, STAGED, WALD, WATERTIGHT, _adjoint, _field, _render, scene_parameters

pytestmark = pytest.mark.gpu

SMALL = 3
HUGE = (1e20, 1e20, 0.5)


def _room(**kw):
    return scenes.room_scene(width=65, height=33, mis=True, box_materials=[scenes.material("diffuse", albedo=HUGE)] * 2, **kw)


def _objects(**kw):
    s = _field(65, 33, **kw)
    for m in s.materials[::3]:
        m.update(scenes.material("diffuse", albedo=HUGE))
    return s


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("film", [KAHAN, LERP])
@pytest.mark.parametrize("make", [_room, _objects, lambda: _room(light="sphere"), lambda: _objects(mis=0)])
def test_films_are_the_megakernels(make, film, isect):
    want = _render(make(), MEGAKERNEL, [1, 2], isect, film, {})
    mean = want[-1][0].view(np.float32)[..., :3]
    assert np.isfinite(mean).all() and (mean > 0).any()
    for route in (STAGED, SMALL):
        got = _render(make(), route, [1, 2], isect, film, {})
        for a, b in zip(want, got):
            assert np.array_equal(a[0], b[0]), route
            assert np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("make", [_room, _objects, lambda: _objects(sky="sun")])
def test_the_adjoint_is_the_replays(make, isect):
    s = make()
    s.render = dict(s.render, spp=3, bounces=5, rr=5)
    params = scene_parameters(s)
    gi = torch.from_numpy(np.random.default_rng(1).normal(size=(33, 65, 3)).astype(np.float32)).cuda()
    img, grads = _adjoint(s, params, gi, isect, STAGED)
    want, want_grads = _adjoint(s, params, gi, isect, MEGAKERNEL)
    assert bool(torch.isfinite(want).all()) and bool((want > 0).any())
    assert torch.equal(img.view(torch.int32), want.view(torch.int32))
