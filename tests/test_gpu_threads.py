"""Contexts on threads of their own, whose scenes need walk stacks of different
sizes, call the same kernels side by side: no call fails, and every film is the
one the context renders alone."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes

from test_gpu_routes import _field

pytestmark = pytest.mark.gpu

ROUNDS = 400


class _Context:
    def __init__(self, s):
        self.s, self.built = s, scenes.BuiltPayload(s)
        self.spec = self.built.default_spec(s.render["bounces"], s.render["bounces"])
        self.camera, self.hosek = scenes.make_camera(s.camera), scenes.make_hosek(s.hosek)
        self.w, self.h = s.camera["w"], s.camera["h"]
        _capi.call("load_cuda_data", C.byref(self.built.payload), C.byref(self.hosek), C.byref(self.camera),
                   C.byref(self.spec), None)

    def film(self, route):
        _capi.call("noor_route", route, 0)
        f = C.c_uint(1)
        _capi.call("cuda_path_tracer", C.byref(f))
        out = np.zeros((self.h, self.w, 4), np.float32)
        _capi.call("noor_get_framebuffer", out.ctypes.data_as(_capi.pf), self.w * self.h)
        return out.view(np.uint32)

    def rays(self, rays, hits):
        _capi.call("noor_trace_closest", C.c_void_p(rays.data_ptr()), C.c_void_p(hits.data_ptr()), rays.shape[0])


def test_stacks_of_different_sizes_side_by_side():
    torch.zeros(1, device="cuda")
    made = [lambda: scenes.room_scene(width=33, height=17, bounces=2), lambda: _field(33, 17, "sun", bounces=2)]
    gate, errors = threading.Barrier(len(made)), []

    def work(make):
        try:
            c = _Context(make())
            rays = torch.zeros((64, 8), device="cuda")
            rays[:, 3], rays[:, 6] = 100.0, 1.0
            hits = torch.zeros((64, 8), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            want = {r: c.film(r) for r in (1, 2, 3)}
            gate.wait(60)
            for k in range(ROUNDS):
                for r in want:
                    if not np.array_equal(c.film(r), want[r]):
                        raise AssertionError("film of route %d" % r)
                c.rays(rays, hits)
            gate.wait(60)
            _capi.call("device_free_memory")
        except BaseException as e:       # noqa: B902
            errors.append(repr(e))
            gate.abort()

    threads = [threading.Thread(target=work, args=(m,)) for m in made]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_builds_of_different_bins_side_by_side():
    torch.zeros(1, device="cuda")
    gate, errors = threading.Barrier(2), []

    def work(bins):
        try:
            s = scenes.SceneData(**scenes.sphere_field(3, 2, 3)[0])
            s.bvh = dict(scenes.DEFAULT_BVH, num_bins=bins)
            want = scenes.BuiltPayload(s, gpu=True).nodes().view(np.uint32).copy()
            gate.wait(60)
            for _ in range(ROUNDS):
                if not np.array_equal(scenes.BuiltPayload(s, gpu=True).nodes().view(np.uint32), want):
                    raise AssertionError("nodes of %d bins" % bins)
        except BaseException as e:       # noqa: B902
            errors.append(repr(e))
            gate.abort()

    threads = [threading.Thread(target=work, args=(b,)) for b in (8, 64)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
