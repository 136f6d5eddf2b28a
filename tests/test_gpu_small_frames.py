"""Frames of few paths: one launch (and the fold of several samples), whatever
the bounce limit, and the megakernel's film to the bit: single paths, sizes
that leave a warp, a block or the pixel tiles unfilled, every count of paths a
warp, both film modes, several samples, films continued, every kernel of the
dispatch, and frames on both sides of the line to the staged renderer."""
import ctypes as C

import numpy as np
import pytest

from noor_b200 import _capi, scenes

from test_gpu_routes import KAHAN, LERP, MEGAKERNEL, WALD, WATERTIGHT, _field, _render
from test_gpu_stages import CASES as STAGE_CASES

pytestmark = pytest.mark.gpu

AUTO, SMALL = 0, 3


def _same(want, got):
    for a, b in zip(want, got):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("isect", [WATERTIGHT, WALD])
@pytest.mark.parametrize("name", list(STAGE_CASES))
def test_every_kind_of_scene(name, isect):
    make, frames = STAGE_CASES[name]
    calls = [min(frames, 20)]
    _same(_render(make(), MEGAKERNEL, calls, isect, KAHAN, {}), _render(make(), SMALL, calls, isect, KAHAN, {}))


@pytest.mark.parametrize("w,h,calls,film", [(1, 1, [1, 1, 1], LERP), (1, 1, [300], KAHAN), (3, 5, [1], KAHAN),
                                            (7, 3, [2, 1], KAHAN), (33, 31, [1, 1], LERP), (49, 48, [1, 3, 1], KAHAN),
                                            (69, 69, [1], KAHAN), (137, 138, [1], KAHAN), (193, 196, [1, 1], KAHAN),
                                            (64, 48, [30], KAHAN), (271, 280, [1], KAHAN), (336, 338, [1], KAHAN),
                                            (337, 338, [1], KAHAN), (389, 390, [1], KAHAN)])
@pytest.mark.parametrize("scene", ["room", "field", "textured"])
def test_every_size(scene, w, h, calls, film):
    make = {"room": lambda: scenes.room_scene(width=w, height=h), "field": lambda: _field(w, h, "sun"),
            "textured": lambda: scenes.textured_room_scene(width=w, height=h)}[scene]
    want = _render(make(), MEGAKERNEL, calls, WATERTIGHT, film, {})
    for route in (AUTO, SMALL):
        _same(want, _render(make(), route, calls, WATERTIGHT, film, {}))


@pytest.mark.parametrize("make", [lambda: scenes.room_scene(width=256, height=256, bounces=64),
                                  lambda: scenes.textured_room_scene(width=192, height=144, bounces=64),
                                  lambda: _field(192, 144, "sun", bounces=64)])
def test_a_small_frame_is_one_launch(make):
    """launches grow with the bounce limit in the stages, not here"""
    r = scenes.Renderer(make())
    try:
        n = [C.c_uint64(), C.c_uint64()]
        r.path_tracer()
        _capi.call("noor_launch_count", C.byref(n[0]))
        r.path_tracer()
        _capi.call("noor_launch_count", C.byref(n[1]))
        assert n[1].value - n[0].value == 1
    finally:
        r.close()
