"""A mesh upload that finds no host memory says so and leaves the scene as it was."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import resource, sys
import numpy as np
sys.path[:0] = [ROOT + "/snake-vk_gb300", ROOT + "/tests"]
import snkpt
from helpers import assert_hits_equal, random_rays
from snkpt import abi, scenes

sc = scenes.config1(width=64, height=36)
pt = snkpt.PathTracer(0)
pt.load_scene(sc)
rays = random_rays(sc, 1000, np.random.default_rng(1))
before = pt.trace_rays(rays)
n = 40_000_000
big = scenes.Mesh(np.zeros((n, 3), np.float32), None, np.zeros((1, 3), np.uint32))
big.positions[:] = 0.0   # (its pages are there before the limit)
now = next(int(l.split()[1]) << 10 for l in open("/proc/self/status") if l.startswith("VmSize"))
soft, hard = resource.getrlimit(resource.RLIMIT_AS)
resource.setrlimit(resource.RLIMIT_AS, (now + (64 << 20), hard))
try:
    pt.upload_meshes([big])
    print("accepted")
except snkpt.SnkError as e:
    print("code", e.code)
resource.setrlimit(resource.RLIMIT_AS, (soft, hard))
pt.set_instances(sc.instances)
pt.build()
assert_hits_equal(pt.trace_rays(rays), before, "the old scene")
pt.load_scene(sc)
assert_hits_equal(pt.trace_rays(rays), before, "loaded again")
print("same")
"""


def test_upload_without_host_memory(cuda, built_lib):
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\n" + CHILD], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["code", "3", "same"], (r.returncode, r.stdout, r.stderr[-2000:])
