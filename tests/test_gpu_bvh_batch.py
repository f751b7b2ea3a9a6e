"""Mesh BVHs built together (all meshes of a scene in one build) against the CPU
oracle and against builds of one mesh at a time."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal, random_rays
from snkpt import scenes

pytestmark = pytest.mark.gpu


def soup(n, rng):
    """n triangles scattered over a unit box, every eighth a copy of the one before (equal Morton codes)."""
    c = rng.uniform(-0.5, 0.5, (n, 1, 3))
    v = (c + rng.normal(0.0, 0.08, (n, 3, 3))).astype(np.float32)
    v[7::8] = v[6::8][:len(v[7::8])]
    return scenes.Mesh(v.reshape(-1, 3), None, np.arange(3 * n, dtype=np.uint32).reshape(n, 3))


def scene_of(meshes, rng):
    rows = [(scenes.affine(scenes.random_rotation(rng), (3.0, 3.0, 3.0), rng.uniform(0.0, 12.0, 3)), k, 0)
            for k in range(len(meshes))]
    mats = scenes.make_materials([((0.5, 0.5, 0.5), 0.5, 0.0, 0)])
    return scenes.Scene(meshes, scenes.make_instances(rows), mats, scenes.no_dir_light(), scenes.point_lights([]))


# tree sizes around the treelet (7), the blocks (256), the sort's chunks (1024) and tiles, and the one-CTA sort (2048)
@pytest.mark.parametrize("sizes", [[1], [2], [7], [8], [2048], [2049], [1, 2, 3, 6, 7, 8, 9, 1], [255, 256, 257, 1],
                                   [1023, 1025, 1, 4096, 2], [1] * 300 + [5] * 40],
                         ids=lambda s: f"{len(s)}x{max(s)}")
@pytest.mark.parametrize("knobs", [{}, {"bvh_treelet_passes": 0xFFFFFFFF, "bvh_leaf_max": 2},
                                   {"bvh_collapse": 1, "bvh_treelet_passes": 0xFFFFFFFF}], ids=["default", "lbvh", "greedy"])
def test_meshes_built_together(cuda, built_lib, sizes, knobs):
    rng = np.random.default_rng(len(sizes) * 1000 + max(sizes))
    meshes = [soup(n, rng) for n in sizes]
    sc = scene_of(meshes, rng)
    pt = snkpt.PathTracer(0)
    pt.set_tuning(knobs)
    pt.load_scene(sc)
    rays = random_rays(sc, 20_000, rng)
    assert_hits_equal(pt.trace_rays(rays), O.OracleScene(sc).trace(rays), str(sizes))
    s = pt.stats()
    assert s["device_error"] == 0 and s["triangles"] == sum(sizes)
    if len(sizes) > 20:
        return
    # the SAH cost is the triangle-weighted mean of the meshes' own trees
    cost = 0.0
    for m in meshes:
        one = snkpt.PathTracer(0)
        one.set_tuning(knobs)
        one.load_scene(scene_of([m], np.random.default_rng(1)))
        cost += one.stats()["blas_sah_cost"] * m.num_triangles / sum(sizes)
    assert s["blas_sah_cost"] == pytest.approx(cost, rel=1e-5)   # (areas and their ratios in binary32)


def test_several_batches(cuda, built_lib):
    """More triangles than one build takes together (2^20), with an empty mesh between."""
    rng = np.random.default_rng(5)
    n = 560
    tiles = [scenes.grid_mesh(n, n, 4.0, 4.0, scenes.value_noise(n, 4, rng)) for _ in range(2)]
    empty = scenes.Mesh(np.zeros((0, 3), np.float32), None, np.zeros((0, 3), np.uint32))
    sc = scene_of([tiles[0], empty, scenes.icosphere(2), tiles[1], scenes.cube_mesh()], rng)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    rays = random_rays(scene_of([tiles[0], scenes.icosphere(2)], rng), 50_000, rng)
    assert_hits_equal(pt.trace_rays(rays), O.OracleScene(sc).trace(rays), "batches")
    assert pt.stats()["triangles"] == 4 * n * n + 320 + 12
