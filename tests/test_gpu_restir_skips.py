"""ReSTIR frames in which many visibility tests can change nothing (no ray is traced for
them): bits and numbers of tests against the CPU oracle over frames with history."""
import numpy as np
import pytest

import oracle as O
import snkpt
from snkpt import abi, scenes
from test_gpu_render import _compare, _gpu_frame

pytestmark = pytest.mark.gpu


def below(sc, share, scale=1.0):
    """The first `share` of the emissive quads under the ground; all radiances times scale."""
    quads = np.flatnonzero(sc.instances["mesh_id"] == len(sc.meshes) - 1)
    sc.instances["transform"][quads[:int(share * len(quads))], 7] = -80.0
    sc.instances["prev_transform"] = sc.instances["transform"]
    sc.materials["albedo"][(sc.materials["flags"] & scenes.MAT_EMISSIVE) != 0] *= np.float32(scale)


def sun_below(sc):
    sc.dir_light["dir"] = -sc.dir_light["dir"]


@pytest.mark.parametrize("case", ["all lights under the ground", "half of them", "sun from below", "strong lights",
                                  "faint lights", "one neighbour, no history"])
def test_tests_that_change_nothing(cuda, built_lib, case):
    W, H, F = 96, 54, 3
    sc = scenes.config2(width=W, height=H, frames=F)
    if case == "sun from below":
        sun_below(sc)
    elif case != "one neighbour, no history":
        below(sc, {"all lights under the ground": 1.0, "half of them": 0.5}.get(case, 0.1),
              {"strong lights": 1e15, "faint lights": 1e-30}.get(case, 1.0))
    knobs = {"restir_temporal": 0, "restir_spatial": 1} if case.startswith("one") else {}
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    ors = O.OracleRestir(O.OracleScene(sc), W, H)
    for f in range(F):
        st = abi.settings(mode=abi.MODE_RESTIR_DI, frame_index=f, seed=3, **knobs)
        g = _gpu_frame(pt, [sc.views[f]], st, cuda)[0]
        ctr = np.zeros(5, np.uint64)
        r, _ = ors.frame(sc.views[f], st, counters=ctr)
        _compare(g, r, f"{case}, frame {f}")
        s = pt.stats()
        assert s["rays_shadow"] + s["shadow_tests_reused"] == int(ctr[2])
        assert s["device_error"] == 0


# entries of the visibility queue are split into slot and pixel: the smallest views and odd numbers of pixels
@pytest.mark.parametrize("W,H,spatial", [(1, 1, 3), (2, 1, 32), (5, 3, 1), (31, 7, 3), (64, 33, 5)])
def test_small_views(cuda, built_lib, W, H, spatial):
    sc = scenes.config2(width=W, height=H, frames=2)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    ors = O.OracleRestir(O.OracleScene(sc), W, H)
    for f in range(2):
        st = abi.settings(mode=abi.MODE_RESTIR_DI, frame_index=f, seed=5, restir_spatial=spatial)
        g = _gpu_frame(pt, [sc.views[f]], st, cuda)[0]
        ctr = np.zeros(5, np.uint64)
        r, _ = ors.frame(sc.views[f], st, counters=ctr)
        _compare(g, r, f"{W}x{H}, frame {f}")
        s = pt.stats()
        assert s["rays_shadow"] + s["shadow_tests_reused"] == int(ctr[2]) and s["device_error"] == 0
