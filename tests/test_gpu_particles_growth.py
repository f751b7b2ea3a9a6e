"""Particle queries on device buffers allocate nothing, neither a context's first one nor those of a
particle system that grows by a few particles per step."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import random_rays
from snkpt import scenes
from test_gpu_particles_parts import DT, PART, bits, particles

pytestmark = pytest.mark.gpu


def test_queries_allocate_nothing(cuda, built_lib):
    import torch
    sc = scenes.config1(width=64, height=36)
    osc = O.OracleScene(sc)
    p = particles(4 * PART, np.random.default_rng(2))
    r = random_rays(sc, 1000, np.random.default_rng(3))
    all_p = torch.from_numpy(p.view(np.float32).reshape(-1, 12).copy()).cuda()
    keep = torch.empty(1 << 30, dtype=torch.uint8, device=cuda)   # (what the outputs below are cut from)
    del keep
    other = snkpt.PathTracer(0)   # loads the kernels
    other.load_scene(sc)
    other.particle_probe(all_p[:1], DT)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(cuda)[0]
    for n in (65_537, 65_600, 80_000, 131_072, 131_073, PART - 1, PART, PART + 1, 4 * PART):
        c, g = pt.particle_probe(all_p[:n], DT)
        at = np.unique([0, n // 2, min(PART, n - 1), n - 1])
        rc, rg = osc.particle_probe(p[at], DT)
        assert np.array_equal(bits(c[at].cpu().numpy()), bits(rc).reshape(len(at), -1))
        assert np.array_equal(bits(g[at].cpu().numpy()), bits(rg))
        assert torch.cuda.mem_get_info(cuda)[0] == free, f"{n} particles"
    # the next build takes the scratch back
    pt.load_scene(sc)
    assert np.array_equal(bits(pt.contact_rays(r, DT)), bits(osc.contact_rays(r, DT)))
