"""Trees of one mesh around the one-block sort's limit (4,096 primitives) with the builder's other forms
(plain LBVH with two primitives per leaf, greedy collapse) against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal, random_rays
from test_gpu_bvh_batch import scene_of, soup

pytestmark = pytest.mark.gpu

LBVH = {"bvh_treelet_passes": 0xFFFFFFFF}


@pytest.mark.parametrize("n", [4096, 4097])
@pytest.mark.parametrize("knobs", [{**LBVH, "bvh_leaf_max": 2}, {**LBVH, "bvh_collapse": 1}], ids=["lbvh", "greedy"])
def test_builder_forms_at_the_sort_line(cuda, built_lib, n, knobs):
    rng = np.random.default_rng(n)
    sc = scene_of([soup(n, rng)], rng)
    pt = snkpt.PathTracer(0)
    pt.set_tuning(knobs)
    pt.load_scene(sc)
    rays = random_rays(sc, 20_000, rng)
    assert_hits_equal(pt.trace_rays(rays), O.OracleScene(sc).trace(rays), f"{n} {knobs}")
    s = pt.stats()
    assert s["device_error"] == 0 and s["triangles"] == n
