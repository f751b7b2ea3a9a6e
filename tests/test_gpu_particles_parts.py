"""Particle queries around the size that one part of a query takes (2^20 rays), and the smallest."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import random_rays
from snkpt import abi, scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0
PART = (1 << 20) // 4   # particles per part of the probe


@pytest.fixture(scope="module")
def world(cuda, built_lib):
    sc = scenes.config1(width=64, height=36)
    pt = snkpt.PathTracer(0)
    pt.load_scene(sc)
    return sc, pt, O.OracleScene(sc)


def particles(n, rng):
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    p["position_radius"][:, :3] = rng.uniform([0.0, 0.0, 0.0], [100.0, 2.0, 100.0], (n, 3))
    p["position_radius"][:, 3] = rng.uniform(0.05, 1.0, n)
    p["velocity"][:, :3] = rng.normal(0.0, 5.0, (n, 3))
    p["velocity"][:, 3] = 1.0
    return p


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("n", [1, 3, PART, PART + 1])
def test_probe_parts(world, n):
    sc, pt, osc = world
    p = particles(n, np.random.default_rng(n))
    c, g = pt.particle_probe(p, DT)
    edge = np.unique(np.clip([0, 1, n // 2, PART - 1, PART, n - 1], 0, n - 1))
    rc, rg = osc.particle_probe(p[edge], DT)
    assert np.array_equal(bits(c[edge]), bits(rc)) and np.array_equal(bits(g[edge]), bits(rg))
    # the same particles asked for in two calls
    k = n // 3
    if k:
        c0, g0 = pt.particle_probe(p[:k], DT)
        c1, g1 = pt.particle_probe(p[k:], DT)
        assert np.array_equal(bits(c), bits(np.concatenate([c0, c1])))
        assert np.array_equal(bits(g), bits(np.concatenate([g0, g1])))


def test_contact_and_constrain_parts(world):
    sc, pt, osc = world
    rng = np.random.default_rng(8)
    n = (1 << 20) + 1
    rays = random_rays(sc, n, rng)
    rays["tmax"] = rng.uniform(0.5, 60.0, n)
    edge = np.array([0, n // 2, n - 2, n - 1])
    assert np.array_equal(bits(pt.contact_rays(rays, DT)[edge]), bits(osc.contact_rays(rays[edge], DT)))
    p = particles(n, rng)
    off = rng.normal(0.0, 0.5, (n, 3)).astype(np.float32)
    off[::7] = 0.0
    assert np.array_equal(bits(pt.particle_constrain(p, off, DT)[edge]),
                          bits(osc.particle_constrain(p[edge], off[edge], DT)))
