"""Instances of meshes whose vertices lie far from the mesh's own origin (baked or georeferenced
parts) and whose transforms bring them back: the roundings of the object-space ray grow with the
vertices' distance, the instances' world boxes must cover them.  Rays that graze an instance at
its outermost vertices hit what the CPU oracle hits."""
import numpy as np
import pytest

import oracle as O
import snkpt
from helpers import assert_hits_equal
from snkpt import abi, scenes

pytestmark = pytest.mark.gpu


def meshes_at(c, rng):
    """A cube, a flat grid tilted a little, and a soup of triangles, moved by c."""
    cube, flat = scenes.cube_mesh(), scenes.grid_mesh(3, 3, 2.0, 2.0, np.zeros((4, 4), np.float32))
    tilt = scenes.rot_x(0.002)
    v = [2.0 * cube.positions.astype(np.float64), flat.positions @ tilt.T, rng.normal(0.0, 0.5, (60, 3))]
    ix = [cube.indices, flat.indices, np.arange(60, dtype=np.uint32).reshape(20, 3)]
    return [scenes.Mesh((p + c).astype(np.float32), None, i) for p, i in zip(v, ix)]


def effective(mesh, transform):
    """World positions (binary64) at which the traversal's binary32 inverse transform sees the vertices."""
    inv = np.asarray(O.invert_affine(transform)[0], np.float64).reshape(3, 4)
    return np.linalg.solve(inv[:, :3], (mesh.positions.astype(np.float64) - inv[:, 3]).T).T


def grazing_rays(sc, rng, per=6):
    rows = []
    for inst in sc.instances:
        m = sc.meshes[int(inst["mesh_id"])]
        w, tri = effective(m, inst["transform"]), np.asarray(m.indices).reshape(-1, 3)
        for axis in range(3):
            for sign in (-1.0, 1.0):
                v = tri.ravel()[np.argmax(sign * w[tri.ravel(), axis])]
                for t in tri[(tri == v).any(1)][:2]:
                    p = np.where(t == v, 0.998, 0.001) @ w[t]
                    for _ in range(per):
                        d = rng.normal(size=3)
                        d[axis] *= 0.02
                        d /= np.linalg.norm(d)
                        rows.append(np.concatenate([p - 6.0 * d, d]))
    rows = np.asarray(rows)
    r = np.zeros(len(rows), abi.RAY_DTYPE)
    r["o"], r["d"], r["tmax"] = rows[:, :3], rows[:, 3:], 1e6
    return r


@pytest.mark.parametrize("far", [0.0, 1e3, 1e4, 1e5, 1e6])
@pytest.mark.parametrize("refit", [0, 4])
def test_grazing_hits_of_far_meshes(cuda, built_lib, far, refit):
    rng = np.random.default_rng(int(far) + refit)
    c = far * np.array([0.8, -0.36, 0.48])
    meshes = meshes_at(c, rng)

    def rows(shift):
        out = []
        for k in range(120):
            R = scenes.rot_x(r[k, 0]) @ scenes.rot_y(r[k, 1]) if k % 2 else scenes.random_rotation(np.random.default_rng(k))
            s = np.array([(1, 1, 1), (2, 1, -1), (0.5, 3, 1)][k % 5 % 3])
            at = 9.0 * np.array([k % 6, k // 6 % 5, k // 30]) + shift
            # minus where the rounded linear part takes the offset: the translation cancels it
            A = scenes.affine(R, s)
            A[:, 3] = at - A[:, :3].astype(np.float64) @ c
            out.append((A, k % 3, 0))
        return out

    r = rng.uniform(-0.004, 0.004, (120, 2))
    mats = scenes.make_materials([((0.5, 0.5, 0.5), 0.5, 0.0, 0)])
    sc = scenes.Scene(meshes, scenes.make_instances(rows(0.0)), mats, scenes.no_dir_light(), scenes.point_lights([]))
    pt = snkpt.PathTracer(0)
    pt.set_tuning({"tlas_refit_interval": refit})
    pt.load_scene(sc)
    if refit:   # new boxes into the old tree
        sc = scenes.Scene(meshes, scenes.make_instances(rows(0.7)), mats, scenes.no_dir_light(), scenes.point_lights([]))
        pt.set_instances(sc.instances)
        pt.build()
    rays = grazing_rays(sc, rng)
    ref = O.OracleScene(sc).trace(rays)
    assert (ref["flags"] == 1).mean() > 0.2
    assert_hits_equal(pt.trace_rays(rays), ref, f"offset {far:g}")
    assert pt.stats()["device_error"] == 0
