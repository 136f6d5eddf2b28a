"""The device payload build (noor_build_payload_gpu) against the host builder,
every payload word the same, where its boxes and its node arrays can go wrong:
meshes at the edges of the 2048-triangle runs whose boxes one block reduces
(the last one short, whole, or of one triangle), coordinates that are zeros of
both signs (a box keeps the first of equal coordinates), meshes without
triangles, and lights whose one-node trees stand before, between and after the
meshes' trees."""
import numpy as np
import pytest

from noor_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(counts, lights, grid, seed):
    rng = np.random.default_rng(seed)
    base = scenes.room_scene(light="sphere")
    tris = int(sum(counts))
    n = max(8, tris // 2)
    V = np.ones((n, 4), np.float32)
    if grid:
        V[:, :3] = rng.choice(np.array([-0.0, 0.0, 1.0, -1.0, 2.0], np.float32), (n, 3))
    else:
        V[:, :3] = rng.normal(0.0, 3.0, (n, 3))
    N = np.zeros((5, 4), np.float32)
    N[:, 1] = 1.0
    meshes, at = [], 0
    for k, c in enumerate(counts):
        if lights and k % 2 == 0:
            meshes.append(dict(tri_start=0, tri_count=0, to_global=scenes.IDENTITY, instance=-1, light_idx=0))
        meshes.append(dict(tri_start=at, tri_count=c, to_global=scenes.IDENTITY, instance=-1, light_idx=-1))
        at += c
    if lights:
        meshes.append(dict(tri_start=0, tri_count=0, to_global=scenes.IDENTITY, instance=-1, light_idx=0))
    return scenes.SceneData(
        vertices=V, normals=N, uvs=rng.random((7, 2)).astype(np.float32),
        vindices=rng.integers(0, n, (tris, 3)).astype(np.uint32),
        nindices=rng.integers(0, 5, (tris, 3)).astype(np.uint32),
        uvindices=rng.integers(0, 7, (tris, 3)).astype(np.uint32),
        material_indices=rng.integers(0, len(base.materials), tris).astype(np.uint32),
        meshes=meshes, materials=base.materials, area_lights=base.area_lights if lights else [], name="edges")


@pytest.mark.parametrize("lights", [False, True])
@pytest.mark.parametrize("counts,grid", [((1,), True), ((2047, 1, 2048), False), ((2049, 4097), False),
                                         ((300, 0, 2048, 0, 5), True), ((70000,), False), ((9000, 3), True)])
def test_boxes_and_node_places(counts, grid, lights):
    scene = _scene(counts, lights, grid, seed=len(counts) + counts[0])
    host, gpu = scenes.BuiltPayload(scene), scenes.BuiltPayload(scene, gpu=True)
    a, b = host.payload, gpu.payload
    assert (a.bvh_root_node, a.num_bvh_nodes, a.num_vertices) == (b.bvh_root_node, b.num_bvh_nodes, b.num_vertices)
    for f in ("num_inner_nodes", "num_leaf_nodes", "height", "max_leaf_tris"):
        assert getattr(host.stat, f) == getattr(gpu.stat, f), f
    assert np.array_equal(host.stat.scene_radius, gpu.stat.scene_radius, equal_nan=True)
    assert host.nodes().view(np.uint32).tolist() == gpu.nodes().view(np.uint32).tolist()
    assert np.array_equal(host.triangle_order(), gpu.triangle_order())
    for name in ("attribute_indices", "wald_ax_nu_nv_nd", "wald_bnu_bnv_au_av", "wald_cnu_cnv_deg_mat"):
        x, y = host.array(name, 4).view(np.uint32), gpu.array(name, 4).view(np.uint32)
        assert np.array_equal(x, y), name
    for name, w in (("vertices", 4), ("normals", 4), ("uvs", 2)):
        x = np.ctypeslib.as_array(getattr(a, name), (a.num_vertices, w)).view(np.uint32)
        y = np.ctypeslib.as_array(getattr(b, name), (b.num_vertices, w)).view(np.uint32)
        assert np.array_equal(x, y), name
