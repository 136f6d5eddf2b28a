"""The staged adjoint at the sizes where its chunks and records can go wrong: a
single pixel, odd sizes, one bounce, a sample count that leaves a remainder in
the last chunk, no environment map.  An image of n samples is the mean of the
n one-sample images, and its gradients the mean of theirs: FP32 sums of the
same terms in another order, good to a few 1e-7 per step of the sum."""
import ctypes as C

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes
from noor_b200.adjoint import _desc, scene_parameters

pytestmark = pytest.mark.gpu


def _step(cam, params, gi, spp, first, bounces):
    alb, rough, env = params
    h, w = cam["h"], cam["w"]
    d = _desc((w, h, spp, first, bounces), alb, rough, env)
    img = torch.zeros((h, w, 3), device="cuda")
    ga, gr = torch.zeros_like(alb), torch.zeros_like(rough)
    ge = torch.zeros_like(env) if env.numel() else None
    torch.cuda.synchronize()
    _capi.call("noor_adjoint_forward", C.byref(d), C.c_void_p(img.data_ptr()))
    _capi.call("noor_adjoint_backward", C.byref(d), C.c_void_p(gi.data_ptr()), C.c_void_p(ga.data_ptr()),
               C.c_void_p(gr.data_ptr()), C.c_void_p(ge.data_ptr()) if ge is not None else None)
    return [img] + [t for t in (ga, gr, ge) if t is not None]


@pytest.mark.parametrize("w,h,spp,bounces,sky", [(1, 1, 1, 1, "map"), (33, 17, 3, 1, "map"), (65, 31, 5, 4, "map"),
                                                 (65, 31, 5, 3, "sun"), (700, 701, 9, 2, "map"),
                                                 (64, 48, 2, 24, "map")])
def test_staged_samples_add_up(w, h, spp, bounces, sky):
    s = scenes.adjoint_scene(seed=5, width=w, height=h, spp=spp, bounces=bounces, count=5, level=3, env_w=64, env_h=32)
    if sky == "sun":
        s.env, s.skydome_type = None, _capi.NOOR_SKY_PHYSICAL
        s.hosek = dict(turbidity=3.0, albedo=0.3, sun_lat=1.0, sun_lon=0.8, solar_scale=250.0, solar_radius_scale=2.0)
    r = scenes.Renderer(s)
    try:
        params = scene_parameters(s)
        gi = torch.from_numpy(np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)).cuda()
        whole = _step(s.camera, params, gi, spp, 1, bounces)
        parts = [_step(s.camera, params, gi, 1, 1 + k, bounces) for k in range(spp)]
        for k, got in enumerate(whole):
            want = sum(p[k].double() for p in parts) / spp
            scale = sum(p[k].double().norm() for p in parts) / spp
            assert torch.isfinite(got).all()
            assert float((got.double() - want).norm()) <= 1e-5 * float(scale) + 1e-12, k
        assert w * h == 1 or all(float(g.abs().sum()) > 0 for g in whole[:2])
        assert r.status(reset=True) == 0
    finally:
        r.close()
