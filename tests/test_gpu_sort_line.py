"""Trees at the line between the one-block and the radix sort of Morton codes, with
equal codes, against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal, random_rays
from snkpt import scenes
from test_gpu_bvh_batch import scene_of, soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2049, 4095, 4096, 4097])
@pytest.mark.parametrize("instances", [False, True], ids=["mesh", "instances"])
def test_sort_line(cuda, built_lib, n, instances):
    rng = np.random.default_rng(n)
    if instances:
        mats = scenes.make_materials([((0.5, 0.5, 0.5), 0.5, 0.0, 0)])
        at = rng.uniform(0.0, 60.0, (n, 3))
        at[5::7] = at[4::7][:len(at[5::7])]   # coincident instances: equal codes
        rows = [(scenes.affine(scenes.random_rotation(rng), (0.5, 0.5, 0.5), p), 0, 0) for p in at]
        sc = scenes.Scene([scenes.cube_mesh()], scenes.make_instances(rows), mats, scenes.no_dir_light(),
                          scenes.point_lights([]))
    else:
        sc = scene_of([soup(n, rng)], rng)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    rays = random_rays(sc, 20_000, rng)
    assert_hits_equal(pt.trace_rays(rays), O.OracleScene(sc).trace(rays), str(n))
    assert pt.stats()["device_error"] == 0
