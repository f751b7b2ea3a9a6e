"""ReSTIR's final test toward a point light when its shorter segment is known to be free: an occluder
at exactly the distance that ends the shorter one blocks the whole segment."""
import numpy as np
import pytest

import oracle as O
import snkpt
from snkpt import abi, scenes
from test_gpu_render import _compare, _gpu_frame

pytestmark = pytest.mark.gpu


def under_a_sheet(y, drop, W, H):
    """A floor, lights at height y and a sheet just under them (one float or `drop`)."""
    sheet = np.nextafter(np.float32(y), np.float32(0.0)) if drop is None else np.float32(y) - np.float32(drop)
    mats = scenes.make_materials([((0.6, 0.6, 0.6), 0.8, 0.0, 0)])
    inst = scenes.make_instances([(scenes.affine(None, (40, 1, 40)), 0, 0),
                                  (scenes.affine(None, (400, 1, 400), (0.0, float(sheet), 0.0)), 0, 0)])
    lights = scenes.point_lights([((float(x), y, float(z)), 0.0, (3e5, 3e5, 3e5)) for x in (-20, -7, 5, 18)
                                  for z in (-16, -3, 9, 21)])
    view = scenes.look_at_view((0.0, 6.0, -14.0), (0.0, 0.0, 2.0), 60.0, W, H)
    return scenes.Scene([scenes.quad_mesh()], inst, mats, scenes.no_dir_light(), lights, [view])


# at 9,000 and 12,000 one float is 0.00098, so that the segments' ends are neighbours and about half of the
# hits on the sheet lie on the shorter one's end; at 300 the sheet lies about 0.001 below, at 2 nothing is there
@pytest.mark.parametrize("y,drop", [(9000.0, None), (12000.0, None), (300.0, None), (300.0, 0.00095), (2.0, 0.002)])
@pytest.mark.parametrize("temporal", [0, 1])
def test_occluder_at_the_shorter_end(cuda, built_lib, y, drop, temporal):
    W, H = 96, 54
    sc = under_a_sheet(y, drop, W, H)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    ors = O.OracleRestir(O.OracleScene(sc), W, H)
    for f in range(3):
        st = abi.settings(mode=abi.MODE_RESTIR_DI, frame_index=f, seed=11, restir_temporal=temporal)
        g = _gpu_frame(pt, [sc.views[0]], st, cuda)[0]
        ctr = np.zeros(5, np.uint64)
        r, _ = ors.frame(sc.views[0], st, counters=ctr)
        _compare(g, r, f"y {y}, frame {f}")
        s = pt.stats()
        assert s["rays_shadow"] + s["shadow_tests_reused"] == int(ctr[2]) and s["device_error"] == 0
