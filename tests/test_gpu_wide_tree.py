"""The four-wide traversals at the forms of a tree and a ray where their words
and box tests change: leaves a word cannot hold, boxes that stick out of their
parents', single-member mesh leaves over identity and other instances, light
nodes, origins with a zero component or far outside the scene, directions
around the smallest the box test takes.  Hits are whole numbers and bits:
equal to the oracle's binary traversal."""
import ctypes as C

import numpy as np
import pytest

from noor_b200 import _capi, scenes
from oracle.oracle import Oracle

from gpu_util import random_rays, trace_any, trace_closest
from test_gpu_trace import _check_closest, _grazing_rays

pytestmark = pytest.mark.gpu


def _scene(which):
    if which.startswith("light_"):
        return scenes.room_scene(light=which[6:])
    if which == "instanced":
        import test_ref_payload as trp
        s = trp.instanced_scene()
    else:
        s = scenes.SceneData(**scenes.sphere_field(7, 16, 4)[0], name=which)
        if which == "big_leaves":     # 1 to 16 triangles a leaf: some beyond a word's 8
            s.bvh = dict(scenes.DEFAULT_BVH, max_height=10, min_leaf_tris=9, max_leaf_tris=16)
    s.camera = dict(eye=(0.0, 2.0, 12.0), look_at=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), fov_deg=60.0, w=32, h=32)
    s.render = dict(spp=1, bounces=4, rr=1, mis=0)
    s.skydome_type = _capi.NOOR_SKY_CONSTANT
    return s


def _stick_out(payload):
    """push the far x bound of some inner nodes' children out of their parents' boxes"""
    n = payload.num_bvh_nodes
    hi = np.ctypeslib.as_array(C.cast(payload.bvh_max_axis_count, C.POINTER(C.c_uint32)), (n, 4))
    lo = np.ctypeslib.as_array(C.cast(payload.bvh_min_right_start, C.POINTER(C.c_uint32)), (n, 4))
    kinds = _capi.LIGHT_NODE_MASK | _capi.MESH_INSTANCE_MASK | _capi.MESH_LEAF_MASK | _capi.TRI_LEAF_MASK
    inner = np.flatnonzero((hi[:, 3] & kinds) == 0)
    rng = np.random.default_rng(1)
    for i in rng.choice(inner, size=max(1, len(inner) // 20), replace=False):
        child = i + 1 if rng.random() < 0.5 else lo[i, 3]
        x = hi[child, 0:1].view(np.float32)
        x += np.float32(rng.uniform(0.05, 2.0))


def _rays(payload, n):
    rng = np.random.default_rng(5)
    v = np.ctypeslib.as_array(C.cast(payload.vertices, C.POINTER(C.c_float)), (payload.num_vertices, 4))[:, :3]
    lo, hi = v.min(0), v.max(0)
    inside = random_rays(rng, n, lo, hi)
    zero = random_rays(rng, n, lo, hi)                       # a zero component in the origin
    zero[np.arange(n), rng.integers(0, 3, n)] = np.where(rng.random(n) < 0.5, np.float32(0.0), np.float32(-0.0))
    far = random_rays(rng, n, lo, hi)                        # from far outside towards the scene
    d = far[:, 4:7].astype(np.float64)
    far[:, :3] = far[:, :3] - d * 10.0 ** rng.uniform(1, 7, (n, 1))
    small = random_rays(rng, n, lo, hi)                      # a component near the box test's smallest
    small[np.arange(n), 4 + rng.integers(0, 3, n)] = 10.0 ** rng.uniform(-22, -15, n) * rng.choice([-1.0, 1.0], n)
    short = random_rays(rng, n, lo, hi)
    short[:, 3] = rng.uniform(-0.5, 2.0, n)                  # extents, some of them negative
    return np.concatenate([inside, zero, far, small, short, _grazing_rays(payload, n, 3),
                           _grazing_rays(payload, n, 4, axis=False)])


WALD, WATERTIGHT = _capi.NOOR_ISECT_REF_WALD, _capi.NOOR_ISECT_WATERTIGHT


# light shapes round as the oracle's only in the Wald mode
@pytest.mark.parametrize("which,isect", [("big_leaves", WALD), ("big_leaves", WATERTIGHT), ("stick_out", WALD),
                                         ("stick_out", WATERTIGHT), ("instanced", WALD), ("instanced", WATERTIGHT),
                                         ("light_sphere", WALD), ("light_disk", WALD)])
def test_wide_traversals_equal_the_binary_walk(which, isect):
    s = _scene(which)
    built = scenes.BuiltPayload(s)
    if which == "stick_out":
        _stick_out(built.payload)
    r = scenes.Renderer(s, built=built, intersector=isect)
    orc = Oracle(r.built.payload, r.spec, r.hosek)
    try:
        rays = _rays(r.built.payload, 20_000)
        want = orc.trace_closest(rays, isect)
        _check_closest(trace_closest(rays), want)
        assert np.array_equal(trace_any(rays), orc.trace_any(rays, isect))
        assert 0.01 < want[:, 6].mean() < 0.99
        assert r.status(reset=True) == 0
    finally:
        orc.close()
        r.close()
