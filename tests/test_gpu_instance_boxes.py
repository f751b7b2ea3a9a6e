"""World boxes of instances (cut to the mesh's extents along 13 axes): rays that graze an
instance at its outermost vertices hit what the CPU oracle hits."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal, random_rays
from snkpt import abi, scenes

pytestmark = pytest.mark.gpu


def forms(rng):
    """Object-to-world matrices: turned by the cube's own angles and by any, mirrored, flattened, sheared, tiny, far."""
    q = np.sqrt(0.5)
    out = [scenes.affine(None, (1, 1, 1)), scenes.affine(None, (-1, 2, 1)),
           scenes.affine([[q, 0, q], [0, 1, 0], [-q, 0, q]], (1, 1, 1)),
           scenes.affine([[0, 0, 1], [1, 0, 0], [0, 1, 0]], (1, -3, 0.5))]
    out += [scenes.affine(scenes.random_rotation(rng), s) for s in
            ((1, 1, 1), (1, 1, -1), (3, 0.01, 1), (1e-3, 1e-3, 1e-3), (0.3, 2, 5), (50, 40, 60))]
    shear = np.zeros((3, 4), np.float32)
    shear[:, :3] = rng.normal(size=(3, 3))
    return out + [shear]


def grazing_rays(sc, rng, per=4):
    """For every instance and every world direction +-x +-y +-z: rays across the direction, through points just
    inside the triangles at the instance's outermost vertex."""
    rows = []
    for inst in sc.instances:
        m = sc.meshes[int(inst["mesh_id"])]
        A = np.asarray(inst["transform"], np.float64).reshape(3, 4)
        w = np.asarray(m.positions, np.float64) @ A[:, :3].T + A[:, 3]
        tri = np.asarray(m.indices).reshape(-1, 3)
        size = np.ptp(w, axis=0).max()
        for axis in range(3):
            for sign in (-1.0, 1.0):
                at = tri[np.isin(tri, tri.ravel()[np.argmax(sign * w[tri.ravel(), axis])]).any(1)][:per]
                for t in at:
                    b = np.where(np.arange(3) == np.argmax(sign * w[t, axis]), 0.998, 0.001)
                    p = b @ w[t]
                    d = rng.normal(size=3)
                    d[axis] *= 0.02
                    d /= np.linalg.norm(d)
                    rows.append(np.concatenate([p - 2.0 * size * d, d]))
    rows = np.asarray(rows)
    r = np.zeros(len(rows), abi.RAY_DTYPE)
    r["o"], r["d"], r["tmin"], r["tmax"] = rows[:, :3], rows[:, 3:], 0.0, 1e6
    return r


def soup(n, rng):
    v = rng.normal(0.0, 0.5, (3 * n, 3)).astype(np.float32) + np.float32(5.0)   # (away from the object's origin)
    return scenes.Mesh(v, None, np.arange(3 * n, dtype=np.uint32).reshape(n, 3))


# extents are reduced by blocks (one mesh in it), warps or single triangles: sizes at those edges
@pytest.mark.parametrize("sizes", [[1], [31, 1, 33, 256], [255, 257, 3, 64, 64], [1] * 70 + [40]],
                         ids=lambda s: f"{len(s)}x{max(s)}")
@pytest.mark.parametrize("refit", [0, 4])
def test_grazing_hits(cuda, built_lib, sizes, refit):
    rng = np.random.default_rng(sum(sizes) + refit)
    flat = scenes.grid_mesh(3, 3, 2.0, 2.0, np.zeros((4, 4), np.float32))
    meshes = [soup(n, rng) for n in sizes] + [scenes.icosphere(2), scenes.cube_mesh(), flat]
    place = forms(rng)
    rows = []
    for k in range(max(len(meshes) + 8, 3 * len(place))):
        A = place[k % len(place)].copy()
        A[:, 3] = rng.uniform(-300.0, 300.0, 3) if k % 3 else rng.uniform(-3.0, 3.0, 3)
        rows.append((A, k % len(meshes), 0))
    mats = scenes.make_materials([((0.5, 0.5, 0.5), 0.5, 0.0, 0)])
    sc = scenes.Scene(meshes, scenes.make_instances(rows), mats, scenes.no_dir_light(), scenes.point_lights([]))
    pt = snkpt.PathTracer(0)
    pt.set_tuning({"tlas_refit_interval": refit})
    pt.load_scene(sc)
    if refit:   # the same instances elsewhere: new boxes into the old tree
        for A, _, _ in rows:
            A[:, 3] += np.float32([1.0, 2.0, 3.0])
        sc = scenes.Scene(meshes, scenes.make_instances(rows), mats, scenes.no_dir_light(), scenes.point_lights([]))
        pt.set_instances(sc.instances)
        pt.build()
    for rays in (grazing_rays(sc, rng), random_rays(sc, 20_000, rng)):
        got = pt.trace_rays(rays)
        assert_hits_equal(got, O.OracleScene(sc).trace(rays), f"{len(rays)} rays")
    assert pt.stats()["device_error"] == 0
