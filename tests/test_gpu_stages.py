"""The staged renderer behind cuda_path_tracer / noor_render_frames against the
plain megakernel (noor_megakernel_batch) on the same frames: one material or
light of each kind, textures, bump and alpha maps, every camera, both triangle
tests, odd sizes, several batches of frames, several chunks of a pixel's
samples.  Both evaluate the same expressions with the same rounding and add
the samples in the same order: the films are equal to the bit, and so are the
rays counted."""
import ctypes as C

import numpy as np
import pytest
import torch

from noor_b200 import _capi, scenes

pytestmark = pytest.mark.gpu

M = scenes.material


def _field(kinds, sky, w, h):
    g, (c, r) = scenes.sphere_field(3, 12, 3, kinds=kinds)
    s = scenes.SceneData(**g, camera=dict(scenes.frame_spheres(c, r, 3, clearance=0.5), w=w, h=h),
                         render=dict(spp=1, bounces=6, rr=1, mis=1))
    s.skydome_type = sky
    if sky == _capi.NOOR_SKY_HDR:
        s.env = scenes.env_map(3, 128, 64, peak=50.0)
    elif sky == _capi.NOOR_SKY_PHYSICAL:
        s.hosek = dict(turbidity=3.0, albedo=0.3, sun_lat=1.0, sun_lon=0.8, solar_scale=250.0, solar_radius_scale=2.0)
    return s


def _boxes(kind, w, h):
    return scenes.room_scene(width=w, height=h, mis=True,
                             box_materials=[M(kind), M("metal", distribution=1, roughness=0.3)])


def _camera(s, **kw):
    s.camera = dict(s.camera, **kw)
    return s


CASES = {
    "room": (lambda: scenes.room_scene(width=67, height=35), 3),
    "one_pixel": (lambda: scenes.room_scene(width=1, height=1), 5),
    "metal_env": (lambda: _field(("metal",), _capi.NOOR_SKY_HDR, 161, 90), 2),
    "glass_sky": (lambda: _field(("glass", "diffuse"), _capi.NOOR_SKY_PHYSICAL, 161, 90), 2),
    "sphere_light": (lambda: scenes.room_scene(width=65, height=33, light="sphere", mis=True), 3),
    "spot_light": (lambda: scenes.room_scene(width=65, height=33, light="spot", mis=True), 3),
    "clearcoat": (lambda: _boxes("clearcoat", 65, 33), 3),
    "roughglass": (lambda: _boxes("roughglass", 65, 33), 3),
    "shadowcatcher": (lambda: _boxes("shadowcatcher", 65, 33), 3),
    "textured": (lambda: scenes.textured_room_scene(width=129, height=71, textured_light=True), 3),
    "textured_few": (lambda: scenes.textured_room_scene(width=100, height=100), 1),         # too few paths
    "textured_enough": (lambda: scenes.textured_room_scene(width=100, height=100), 2),
    "lens": (lambda: _camera(scenes.room_scene(width=64, height=36), lens_radius=0.1, focal_length=3.0), 2),
    "env_camera": (lambda: _camera(scenes.room_scene(width=64, height=36), type="env"), 2),
    "batches": (lambda: scenes.room_scene(width=1500, height=1501, bounces=2), 3),         # one frame a batch
    "chunks": (lambda: scenes.room_scene(width=64, height=48, bounces=2), 1400),            # 50 chunks, two batches
}


@pytest.mark.parametrize("isect", [_capi.NOOR_ISECT_WATERTIGHT, _capi.NOOR_ISECT_REF_WALD])
@pytest.mark.parametrize("name", list(CASES))
def test_staged_film_is_the_megakernels(name, isect):
    make, frames = CASES[name]
    s = make()
    w, h = s.camera["w"], s.camera["h"]
    r = scenes.Renderer(s, intersector=isect)
    try:
        r.counters(reset=True)
        r.render(frames)
        got, rays = r.framebuffer(), r.counters(reset=True)
        film = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        f = scenes.wf_frame(0, s.camera, frames, s.render["bounces"], d_film=film.data_ptr())
        _capi.call("noor_megakernel_batch", C.byref(f), 1, None)
        want = film.cpu().numpy()
        assert rays == r.counters(reset=True)
        assert np.isfinite(want).all() and (name == "one_pixel" or want[..., :3].mean() > 0.005)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        assert r.status(reset=True) == 0
    finally:
        r.close()
