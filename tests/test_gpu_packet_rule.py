"""Sizes around the line from which a view's camera rays are traced in warp packets: every
output bit for bit as ray by ray (a lowered step cap turns the packets off)."""
import numpy as np
import pytest

import snkpt
from snkpt import abi, scenes
from test_gpu_render import _gpu_frame

pytestmark = pytest.mark.gpu


def few_triangles(w, h):
    sc = scenes.config0(width=w, height=h)
    keep = sc.instances["mesh_id"] != 0   # without the sphere: 72 triangles
    sc.instances = sc.instances[keep].copy()
    return sc


# the room's line is at 1200 sqrt(2120) = 55,253 rays, few triangles' at 32,768
@pytest.mark.parametrize("room,w,h,spp", [(True, 256, 212, 1), (True, 256, 216, 1), (True, 128, 108, 4), (True, 8, 6912, 1),
                                          (False, 256, 124, 1), (False, 256, 128, 1), (False, 255, 132, 1),
                                          (False, 128, 86, 3)])
def test_packets_around_the_line(cuda, built_lib, room, w, h, spp):
    sc = scenes.config0(width=w, height=h) if room else few_triangles(w, h)
    st = abi.settings(spp=spp, max_depth=3, rr_depth=2, seed=4)
    outs = []
    for knobs in ({}, {"max_traversal_steps": 65535}):
        pt = snkpt.PathTracer(0)
        pt.set_tuning(knobs)
        pt.load_scene(sc)
        outs.append(_gpu_frame(pt, [sc.views[0]], st, cuda)[0])
        assert pt.stats()["device_error"] == 0
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k]), k
    assert (outs[0]["inst_id"] != 0xFFFFFFFF).mean() > 0.3
