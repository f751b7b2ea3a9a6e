"""Few rays: queues too small to fill the GPU, whose rays get eight lanes each, against
the CPU oracle (closest hits bit for bit, any hits), also with deep stacks and with the
traversal's limits."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal, camera_rays, random_rays, shadow_rays
from snkpt import abi, scenes

pytestmark = pytest.mark.gpu


def nested(rng):
    """Shells inside shells: every ray's boxes overlap, so its stack grows past the shared entries."""
    rows = [(scenes.affine(scenes.random_rotation(rng), (s, s, s), rng.normal(0.0, 0.3, 3)), 0, 0)
            for s in np.linspace(0.2, 12.0, 700)]
    mats = scenes.make_materials([((0.5, 0.5, 0.5), 0.5, 0.0, 0)])
    return scenes.Scene([scenes.icosphere(2)], scenes.make_instances(rows), mats, scenes.no_dir_light(),
                        scenes.point_lights([]))


@pytest.fixture(scope="module")
def worlds(cuda, built_lib):
    out = {}
    for name, sc in (("field", scenes.config1(width=64, height=36)), ("nested", nested(np.random.default_rng(3)))):
        pt = snkpt.PathTracer(0)
        pt.load_scene(sc)
        out[name] = sc, pt, O.OracleScene(sc)
    return out


# up to 4 rays per resident warp (24 warps per SM) take the eight-lane path from the start
@pytest.mark.parametrize("n", [1, 2, 5, 33, 1000, "warps", "warps+1", "4 warps", "4 warps+1"])
@pytest.mark.parametrize("world", ["field", "nested"])
def test_few_rays_match_oracle(worlds, n, world):
    import torch
    sc, pt, osc = worlds[world]
    w = 24 * torch.cuda.get_device_properties(0).multi_processor_count
    n = {"warps": w, "warps+1": w + 1, "4 warps": 4 * w, "4 warps+1": 4 * w + 1}.get(n, n)
    rng = np.random.default_rng(n)
    rays = random_rays(sc, n, rng)
    assert_hits_equal(pt.trace_rays(rays), osc.trace(rays), f"{n} closest")
    rays = shadow_rays(sc, n, rng)
    assert np.array_equal(pt.trace_rays(rays, any_hit=True)["flags"], osc.trace(rays, any_hit=True)["flags"])


@pytest.mark.parametrize("width,height", [(1, 1), (9, 5), (64, 36), (160, 90)])
def test_small_frames_match_oracle(worlds, width, height):
    sc = scenes.config1(width=width, height=height)
    _, pt, osc = worlds["field"]
    st = abi.settings(spp=1, max_depth=4, rr_depth=3, seed=9)
    out = snkpt.alloc_outputs(width, height, device="cuda:0")
    pt.render([sc.views[0]], st, [out])
    pt.synchronize()
    ref = osc.render_path(sc.views[0], st)
    g = out["radiance"].cpu().numpy()[:, :3].astype(np.float64)
    r = ref["radiance"][:, :3].astype(np.float64)
    assert float((np.abs(g - r) / np.maximum(np.abs(r), 1e-6)).max()) <= 1e-4
    assert np.array_equal(out["depth"].cpu().numpy(), ref["depth"])


@pytest.mark.parametrize("knob", ["max_traversal_steps", "stack_limit"])
def test_limits_reported_and_recovered(worlds, knob):
    sc, pt, osc = worlds["nested"]
    rays = random_rays(sc, 5, np.random.default_rng(1))
    pt.set_tuning({knob: 1})
    with pytest.raises(snkpt.SnkError) as e:
        pt.trace_rays(rays)
    assert e.value.code == abi.ERR_LIMIT
    pt.set_tuning({})
    assert_hits_equal(pt.trace_rays(rays), osc.trace(rays), "after the limit")
