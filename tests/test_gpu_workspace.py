"""Device memory of the staged renderer and the adjoint: with less than a whole
batch or chunk takes, by the context's limit or because the device has no more,
they take fewer frames or samples at a time, to the same bits, and only where
one does not fit the kernels that need none."""
import ctypes as C

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes
from noor_b200.adjoint import _desc, scene_parameters

pytestmark = pytest.mark.gpu

STAGED = 2


def _launches():
    n = C.c_uint64()
    _capi.call("noor_launch_count", C.byref(n))
    return n.value


def _limit(n):
    _capi.call("noor_workspace_limit", C.c_size_t(n))


def _film(r, frames):
    r.frame = C.c_uint(1)
    at = _launches()
    r.render(frames)
    n = _launches() - at
    return r.framebuffer().view(np.uint32), n


@pytest.mark.parametrize("make,path_bytes", [(lambda: scenes.room_scene(width=203, height=151), 228),
                                             (lambda: scenes.textured_room_scene(width=203, height=151), 292)])
def test_fewer_frames_a_batch(make, path_bytes):
    s = make()
    r = scenes.Renderer(s)
    try:
        _capi.call("noor_route", STAGED, 0)
        frame = 203 * 151 * path_bytes
        want, whole = _film(r, 9)
        batch = 4 + 2 * s.render["bounces"]                     # launches of a batch, and its fold
        assert whole == batch
        # nine frames, halved until they fit: four (three batches), two (five), one (nine)
        for room, batches in ((8.5, 3), (4.5, 3), (2.5, 5), (1.5, 9)):
            _limit(int(room * frame))
            got, n = _film(r, 9)
            assert np.array_equal(got, want) and n == batches * batch, room
        _limit(int(0.5 * frame))
        got, n = _film(r, 9)
        assert np.array_equal(got, want) and n <= 2             # the megakernel and its fold
        _limit(1 << 40)
        got, n = _film(r, 9)
        assert np.array_equal(got, want) and n == whole
    finally:
        r.close()


def test_fewer_samples_a_chunk():
    w, h, spp, bounces = 65, 31, 9, 3
    s = scenes.adjoint_scene(seed=5, width=w, height=h, spp=spp, bounces=bounces, count=5, level=3, env_w=64, env_h=32)
    r = scenes.Renderer(s)
    alb, rough, env = scene_parameters(s)
    gi = torch.from_numpy(np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)).cuda()

    def step():
        d = _desc((w, h, spp, 1, bounces), alb, rough, env)
        img = torch.zeros((h, w, 3), device="cuda")
        g = [torch.zeros_like(t) for t in (alb, rough, env)]
        torch.cuda.synchronize()
        at = _launches()
        _capi.call("noor_adjoint_forward", C.byref(d), C.c_void_p(img.data_ptr()))
        mid = _launches()
        _capi.call("noor_adjoint_backward", C.byref(d), C.c_void_p(gi.data_ptr()), *[C.c_void_p(t.data_ptr()) for t in g])
        return img, g, mid - at, _launches() - mid

    try:
        img, grads, fwd, bwd = step()
        sample = w * h * (184 + 148 * bounces)
        # nine samples, halved until they fit: four (three chunks), two (five), one (nine)
        for room, chunks in ((8.5, 3), (2.5, 5), (1.5, 9)):
            _limit(int(room * sample))
            got, g, f, b = step()
            assert torch.equal(got.view(torch.int32), img.view(torch.int32))
            assert b == chunks * bwd
            for x, y in zip(g, grads):
                assert float((x - y).norm()) <= 1e-5 * float(y.norm())
        _limit(0)                                               # the replay, which needs its own 16 bytes a path
        got, g, f, b = step()
        assert torch.equal(got.view(torch.int32), img.view(torch.int32))
        assert b == 2 * 3                                       # two kernels per four samples
        for x, y in zip(g, grads):
            assert float((x - y).norm()) <= 1e-5 * float(y.norm())
    finally:
        r.close()


def test_a_full_device():
    """some 700 MB free: four 1024x1024 frames (0.96 GB) go in smaller batches"""
    s = scenes.room_scene(width=1024, height=1024, bounces=3)
    r = scenes.Renderer(s)
    hold = []
    try:
        _capi.call("noor_route", STAGED, 0)
        r.render(1)
        want, whole = _film(r, 4)
        _limit(0)                                               # gives the buffer back
        _limit(1 << 40)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        while True:
            free = torch.cuda.mem_get_info()[0]
            take = min(free - (700 << 20), 16 << 30)
            if take < (64 << 20):
                break
            hold.append(torch.empty(take, dtype=torch.uint8, device="cuda"))
        got, n = _film(r, 4)
        assert np.array_equal(got, want)
        assert n > whole                                        # staged, in more batches
        assert r.status(reset=True) == 0
    finally:
        hold.clear()
        torch.cuda.empty_cache()
        r.close()


POOL = r"""
import ctypes as C, sys
import torch
from noor_b200 import _capi, scenes
torch.zeros(1, device="cuda")
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0] >> 20)[1]
make = lambda: scenes.Renderer(scenes.room_scene(width=1024, height=1024))
r = make(); r.close()
at = [free()]
r = make(); r.render(1); r.close()
at.append(free())                      # the next context's: some 240 MB
r = make(); r.render(1)
_capi.call("noor_workspace_limit", C.c_size_t(0))
r.close()
at.append(free())
print(*at)
"""


def test_the_pool_keeps_and_gives_back():
    """host-built payloads only: what a context gives back serves the next one, until it is asked for"""
    import subprocess
    import sys
    from pathlib import Path
    out = subprocess.run([sys.executable, "-c", POOL], capture_output=True, text=True, timeout=300,
                         cwd=Path(__file__).resolve().parents[1])
    assert out.returncode == 0, out.stderr[-2000:]
    before, kept, after = map(int, out.stdout.split())
    assert before - kept >= 200
    assert before - after <= 64
