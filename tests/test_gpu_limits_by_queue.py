"""The traversal's limits (snk_tuning's max_traversal_steps and stack_limit) mean the same for a ray
alone, in a small queue and at the end of a large one: it is reported in all of them or in none."""
import numpy as np
import pytest

import snkpt
from helpers import random_rays
from snkpt import abi
from test_gpu_trace_few import nested

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(cuda, built_lib):
    sc = nested(np.random.default_rng(3))
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    return sc, pt


def reported(pt, ray, n, any_hit):
    """Whether the query of n - 1 empty rays (one step each) and this one is refused."""
    rays = np.repeat(ray, n)
    rays["tmax"][:-1] = -1.0
    try:
        pt.trace_rays(rays, any_hit=any_hit)
    except snkpt.SnkError as e:
        assert e.code == abi.ERR_LIMIT
        return True
    return False


# (20,000 rays are more than four for each of the GPU's warps; the last ray works alone, whatever the queue's size)
@pytest.mark.parametrize("knob,caps", [("max_traversal_steps", [2, 5, 10, 20, 30, 40, 60, 80, 100, 120, 160, 240, 400]),
                                       ("stack_limit", [1, 2, 3, 4, 5, 6, 8, 10, 14, 20])])
@pytest.mark.parametrize("any_hit", [False, True])
def test_same_limit_for_every_queue(world, knob, caps, any_hit):
    sc, pt = world
    seen = set()
    try:
        for ray in random_rays(sc, 12, np.random.default_rng(4)).reshape(-1, 1):
            for cap in caps:
                pt.set_tuning({knob: cap})
                got = [reported(pt, ray, n, any_hit) for n in (1, 64, 20_000)]
                assert got[0] == got[1] == got[2], f"{knob} {cap}: {got}"
                seen.add(got[0])
    finally:
        pt.set_tuning({})
    assert seen == {True, False}
