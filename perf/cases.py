"""What the performance of this path-tracing core is measured on.

Each case is one thing a program built on ``snkpt`` does over and over: render
a frame (plain path tracing, several views at once, ReSTIR, the radiance
cache, an animated scene), load a scene, ask for ray hits or particle contacts,
resolve a frame in time.  Scenes are the seeded generators of ``snkpt.scenes``.

Library work is issued on a stream of its own; ``run`` makes torch's current
stream wait for it, so that the returned tensors can be used there.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "snake-vk_gb300"))

import snkpt  # noqa: E402
from snkpt import abi, scenes  # noqa: E402

DT = 1.0 / 120.0


def listed():
    return [
        # the smallest frame: a preview or thumbnail of a closed room with every output (launches and latency count)
        {"name": "path_room_256", "kind": "path", "scene": "room", "width": 256, "height": 256, "views": 1, "spp": 1,
         "depth": 4, "outputs": "all"},
        # the ordinary frame: 1080p, one sample, four segments, with the G-buffer that a denoiser or TAA takes
        {"name": "path_field_1080", "kind": "path", "scene": "field", "width": 1920, "height": 1080, "views": 1,
         "spp": 1, "depth": 4, "outputs": "all"},
        # the largest frame: the uneven 8-view batch of the terrain (19.2 Mpx, 6 segments), radiance only
        {"name": "path_terrain_batch", "kind": "path", "scene": "terrain", "width": 3840, "height": 2160, "views": 8,
         "spp": 1, "depth": 6, "outputs": "radiance"},
        # an animated scene: every instance moves, the instance tables and BVH are redone, the image goes to the host
        {"name": "animated_quads_720", "kind": "animated", "quads": 4096, "width": 1280, "height": 720, "depth": 3},
        # the render pass as the engine drives it: ReSTIR + indirect light, a first frame and one with history
        {"name": "restir_field_1080", "kind": "restir", "width": 1920, "height": 1080, "spatial": 3, "mode": "pt"},
        # a frame with the radiance cache, which trains its network with four Adam steps
        {"name": "cache_terrain_1080", "kind": "cache", "width": 1920, "height": 1080, "train_paths": 16384},
        # loading a level whose geometry is one large mesh and a small one
        {"name": "load_terrain", "kind": "load", "grid": 256, "parts": 0},
        # loading a model of many submeshes, one BVH each
        {"name": "load_parts_48", "kind": "load", "grid": 32, "parts": 48},
        # line-of-sight tests of a simulation, rays and results on the device
        {"name": "sight_1m", "kind": "rays", "rays": 1 << 20, "any_hit": True, "memory": "device"},
        # a picking query: a handful of closest-hit rays from the host (the smallest call)
        {"name": "pick_64", "kind": "rays", "rays": 64, "any_hit": False, "memory": "host"},
        # one step of a particle system's scene collisions
        {"name": "particles_100k", "kind": "particles", "particles": 100_000},
        # temporal anti-aliasing of two successive frames
        {"name": "taa_1080", "kind": "taa", "width": 1920, "height": 1080},
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["path", "path", "path", "animated", "restir", "cache", "load", "load", "rays", "rays",
                       "particles", "taa"])
    if kind == "path":
        w = _log(rng, 64, 1920)
        h = max(16, min(1080, int(w * rng.uniform(0.4, 1.0))))
        views = rng.choice([1, 1, 1, 2, 5])
        spp = rng.choice([1, 1, 2, 4])
        if w * h * views * spp > 6_000_000:
            views, spp = 1, 1
        return {"kind": kind, "scene": rng.choice(["room", "field", "terrain"]), "width": w, "height": h,
                "views": views, "spp": spp, "depth": rng.randint(2, 6), "outputs": rng.choice(["all", "radiance"])}
    if kind == "animated":
        w = _log(rng, 160, 1920)
        return {"kind": kind, "quads": _log(rng, 16, 4096), "width": w, "height": max(16, w * 9 // 16),
                "depth": rng.randint(1, 4)}
    if kind == "restir":
        w = _log(rng, 160, 1920)
        return {"kind": kind, "width": w, "height": max(16, w * 9 // 16), "spatial": rng.randint(0, 5),
                "mode": rng.choice(["di", "pt"])}
    if kind == "cache":
        w = _log(rng, 320, 1920)
        return {"kind": kind, "width": w, "height": max(16, w * 9 // 16), "train_paths": _log(rng, 1000, 16384)}
    if kind == "load":
        return {"kind": kind, "grid": _log(rng, 8, 400), "parts": rng.choice([0, 1, _log(rng, 2, 48)])}
    if kind == "rays":
        memory = rng.choice(["device", "host"])
        return {"kind": kind, "rays": _log(rng, 1000, 2_000_000) if memory == "device" else _log(rng, 1, 100_000),
                "any_hit": rng.choice([False, True]), "memory": memory}
    if kind == "particles":
        return {"kind": kind, "particles": _log(rng, 100, 500_000)}
    w = _log(rng, 64, 3840)
    return {"kind": "taa", "width": w, "height": max(16, min(2160, int(w * rng.uniform(0.4, 1.0))))}


# ---- inputs -------------------------------------------------------------------
def _scene(case, seed):
    """The scene of a path-traced case and its views."""
    w, h, views = case["width"], case["height"], case["views"]
    if case["scene"] == "terrain" and views == 8:
        return scenes.config3(seed, resolutions=[(max(1, a * w // 3840), max(1, b * h // 2160))
                                                 for a, b in scenes.CONFIG3_RESOLUTIONS])
    if case["scene"] == "terrain":
        return scenes.config3(seed, resolutions=[(max(8, w >> (k % 3)), max(8, h >> (k % 3))) for k in range(views)])
    if case["scene"] == "room":
        sc = scenes.config0(seed, w, h)
        eye, step = np.array([0.0, 5.0, -4.8]), np.array([0.3, -0.2, 0.1])
        target = np.array([0.0, 3.5, 5.0])
    else:
        sc = scenes.config1(seed, w, h)
        eye, step = np.array([50.0, 45.0, -55.0]), np.array([6.0, -2.0, 3.0])
        target = np.array([50.0, 15.0, 50.0])
    sc.views = [scenes.look_at_view(eye + k * step, target, 60.0, max(8, w >> (k % 3)), max(8, h >> (k % 3)))
                for k in range(views)]
    return sc


def _parts(case, rng):
    """A model of `parts` submeshes: icospheres, cubes and small grids of uneven sizes."""
    kinds = [scenes.icosphere(1), scenes.icosphere(2), scenes.icosphere(3), scenes.cube_mesh()]
    out = []
    for k in range(case["parts"]):
        n = int(rng.integers(2, 48))
        out.append(kinds[k % 5] if k % 5 < 4 else
                   scenes.grid_mesh(n, n, 4.0, 4.0, scenes.value_noise(n, 3, rng) * 0.5))
    return out


def _sphere_scene(seed):
    sc = scenes.config1(seed, 64, 36)
    rng = np.random.default_rng(seed)
    prev = sc.instances["transform"].reshape(-1, 3, 4).copy()
    prev[:, :, 3] -= rng.normal(0.0, 0.05, (len(prev), 3)).astype(np.float32)   # the instances moved since last frame
    sc.instances["prev_transform"] = prev.reshape(-1, 12)
    return sc


def _rays(case, rng):
    """Rays between random points of the sphere field (any hit) or from the camera side into it."""
    n = case["rays"]
    r = np.zeros(n, abi.RAY_DTYPE)
    a, b = rng.uniform(0.0, 100.0, (n, 3)), rng.uniform(0.0, 100.0, (n, 3))
    if not case["any_hit"]:
        a = np.array([50.0, 45.0, -55.0]) + rng.normal(0.0, 1.0, (n, 3))
    d = b - a
    dist = np.linalg.norm(d, axis=1, keepdims=True)
    r["o"], r["d"] = a, d / dist
    r["tmin"], r["tmax"] = 0.001, dist[:, 0] if case["any_hit"] else 1e4
    return r


def _particles(sc, n, rng):
    """Particles resting on or flying near the ground and the spheres, some asleep, some still."""
    M = sc.instances["transform"].reshape(-1, 3, 4)
    k = rng.integers(0, 200, n)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rad = np.linalg.norm(M[k, :, 0], axis=1)
    pos = M[k, :, 3] + d * (rad + rng.uniform(0.0, 0.6, n))[:, None]
    ground = rng.uniform(size=n) < 0.4
    pos[ground] = rng.uniform([0.0, 0.0, 0.0], [100.0, 0.6, 100.0], (int(ground.sum()), 3))
    p = np.zeros(n, abi.PARTICLE_DTYPE)
    p["position_radius"][:, :3] = pos
    p["position_radius"][:, 3] = rng.uniform(0.05, 0.5, n)
    v = rng.normal(0.0, 3.0, (n, 3))
    v[rng.uniform(size=n) < 0.05] = 0.0
    p["velocity"][:, :3] = v
    p["velocity"][:, 3] = rng.uniform(size=n) < 0.9
    return p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "taa":
        w, h = case["width"], case["height"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["frames"] = []
        for _ in range(2):
            rad = torch.exp(torch.randn(h * w, 4, generator=g, device="cuda") * 1.2 - 0.5)
            rad[:, 3] = 1.0
            # a moving camera's motion vectors: one smooth field, a few disoccluded pixels
            mot = torch.randn(h * w, 2, generator=g, device="cuda") * 0.0005 + torch.rand(2, generator=g, device="cuda") * 0.01
            far = torch.rand(h * w, 1, generator=g, device="cuda") < 0.02
            st["frames"].append((rad, torch.where(far, mot * 30.0, mot)))
        st["stream"] = torch.cuda.Stream()
        st["taa"] = snkpt.TaaResolve(w, h, stream=st["stream"])
        return st
    st["stream"] = torch.cuda.Stream()
    if kind == "restir":
        st["rt"] = snkpt.RT(0, stream=st["stream"])
        sc = scenes.config2(seed, case["width"], case["height"], frames=2)
        st["rt"].init(sc)
        st["views"] = sc.views
        names = ("radiance", "albedo", "normal", "motion", "depth")
        st["outs"] = [snkpt.alloc_outputs(case["width"], case["height"], "cuda", names) for _ in sc.views]
        st["mode"] = abi.MODE_RESTIR_PT if case["mode"] == "pt" else abi.MODE_RESTIR_DI
        return st
    pt = st["pt"] = snkpt.PathTracer(0, stream=st["stream"])
    if kind == "path":
        sc = _scene(case, seed)
        pt.load_scene(sc)
        st["views"] = sc.views
        names = snkpt.OUTPUT_NAMES if case["outputs"] == "all" else ("radiance",)
        st["outs"] = [snkpt.alloc_outputs(int(v["width"]), int(v["height"]), "cuda", names) for v in sc.views]
        st["settings"] = abi.settings(spp=case["spp"], max_depth=case["depth"], rr_depth=3, seed=seed & 0x7FFFFFFF)
    elif kind == "animated":
        sc = scenes.config2(seed, case["width"], case["height"], frames=2)
        sc.instances = sc.instances[:201 + case["quads"]].copy()
        pt.load_scene(sc)
        st["views"], st["poses"], st["outs"] = sc.views, [], []
        for _ in sc.views:
            inst = sc.instances.copy()
            inst["transform"][:, [3, 7, 11]] += rng.normal(0.0, 0.2, (len(inst), 3)).astype(np.float32)
            st["poses"].append(inst)
            img = torch.empty(case["width"] * case["height"], 4, pin_memory=True)
            st["outs"].append({"radiance": img.numpy()})
            st.setdefault("keep", []).append(img)
        st["settings"] = abi.settings(max_depth=case["depth"], rr_depth=3, seed=seed & 0x7FFFFFFF)
    elif kind == "cache":
        sc = scenes.config4(seed, case["width"], case["height"], frames=8)
        pt.load_scene(sc)
        st["view"] = sc.views[3]
        bound = np.full(snkpt.CACHE_NUM_WEIGHTS, math.sqrt(6.0 / 64.0))
        bound[4 * 4096:] *= 0.1
        st["weights"] = (rng.uniform(-1.0, 1.0, snkpt.CACHE_NUM_WEIGHTS) * bound).astype(np.float32)
        st["out"] = snkpt.alloc_outputs(case["width"], case["height"], "cuda", ("radiance",))
        st["settings"] = abi.settings(mode=abi.MODE_PATH_CACHE, max_depth=6, rr_depth=3, seed=seed & 0x7FFFFFFF,
                                      cache_train_paths=case["train_paths"])
    elif kind == "load":
        sc = scenes.config3(seed, resolutions=[(320, 180)])
        g = case["grid"]
        sc.meshes = [sc.meshes[0], scenes.terrain_tile(rng, g)] + _parts(case, rng)
        for k in range(case["parts"]):   # each part stands somewhere over the terrain
            sc.instances["mesh_id"][k] = 2 + k
        v = sc.views[0]
        x, y = rng.uniform(-1.0, 1.0, (2, 65536))
        t = float(v["tan_half_fov_y"])
        d = v["forward"] + v["right"] * (x * t * float(v["aspect"]))[:, None] + v["up"] * (y * t)[:, None]
        rays = np.zeros(65536, abi.RAY_DTYPE)
        rays["o"], rays["d"], rays["tmax"] = v["pos"], d / np.linalg.norm(d, axis=1, keepdims=True), 1e4
        st["scene"] = sc
        st["rays"] = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    elif kind == "rays":
        st["scene"] = _sphere_scene(seed)
        pt.load_scene(st["scene"])
        r = _rays(case, rng)
        st["rays"] = r if case["memory"] == "host" else torch.from_numpy(r.view(np.float32).reshape(-1, 8).copy()).cuda()
    else:
        sc = _sphere_scene(seed)
        pt.load_scene(sc)
        p = _particles(sc, case["particles"], rng)
        st["particles"] = torch.from_numpy(p.view(np.float32).reshape(-1, 12).copy()).cuda()
    return st


# ---- one pass -------------------------------------------------------------------
def _hits(h):
    """The fields of a hit array, whichever side it is on."""
    if isinstance(h, torch.Tensor):
        f = h.view(torch.float32)
        return {"t": f[:, 0], "u": f[:, 3], "v": f[:, 4], "inst": h[:, 1], "prim": h[:, 2], "flags": h[:, 5]}
    return {k: h[k] for k in ("t", "u", "v", "inst", "prim", "flags")}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    pt = state.get("pt")
    if kind == "path":
        pt.render(state["views"], state["settings"], state["outs"])
        out = state["outs"]
    elif kind == "animated":
        for view, pose, img in zip(state["views"], state["poses"], state["outs"]):
            pt.set_instances(pose)
            pt.build()
            pt.render([view], state["settings"], [img])
        return [o["radiance"] for o in state["outs"]]
    elif kind == "restir":
        rt = state["rt"]
        rt.frame_index = 0
        settings = snkpt.RT.RtSettings(1, case["spatial"])
        for view, o in zip(state["views"], state["outs"]):   # (the first view's history is marked invalid)
            rt.record_render([view], [o], settings, mode=state["mode"])
        out = state["outs"]
    elif kind == "cache":
        pt.cache_set_weights(state["weights"])
        pt.render([state["view"]], state["settings"], [state["out"]])
        out = [state["out"]["radiance"], pt.cache_get_weights()]
    elif kind == "load":
        pt.load_scene(state["scene"])
        out = _hits(pt.trace_rays(state["rays"]))
    elif kind == "rays":
        out = _hits(pt.trace_rays(state["rays"], any_hit=case["any_hit"]))
    elif kind == "particles":
        out = pt.particle_probe(state["particles"], DT)
    else:
        state["taa"].reset()
        out = [state["taa"].resolve(rad, mot) for rad, mot in state["frames"]]
    torch.cuda.current_stream().wait_stream(state["stream"])
    return out


# ---- what a pass cannot do without ------------------------------------------------
RAY_FLOPS = 1700.0          # about 8 wide nodes of 8 boxes, a triangle or two, shading
RAYS_PER_PATH = {"room": 1.4, "field": 0.75, "terrain": 0.6}   # rays (of all kinds) per path and segment
SCENE_BYTES = {"room": 0.3e6, "field": 16e6, "terrain": 16e6}  # nodes, triangles and vertices, read once
OUTPUT_BYTES = {"all": 104, "radiance": 16}


def work(case):
    kind = case["kind"]
    if kind == "path":
        px = sum(int(v["width"]) * int(v["height"]) for v in _views_only(case))
        return {"bytes": px * OUTPUT_BYTES[case["outputs"]] + SCENE_BYTES[case["scene"]],
                "flops": px * case["spp"] * case["depth"] * RAYS_PER_PATH[case["scene"]] * RAY_FLOPS}
    if kind == "taa":
        px = case["width"] * case["height"]
        # per frame 16 + 8 in, 16 + 8 of history in, 16 out, 16 + 8 of the next history out
        return {"bytes": 2 * px * 88.0, "flops": 2 * px * 300.0}
    if kind == "load":
        tris = 2 * case["grid"] ** 2 + 1280 + case["parts"] * 1100
        return {"bytes": tris * (18 + 12 + 48 + 20) + 65536 * 56.0, "flops": tris * 500.0 + 65536 * RAY_FLOPS}
    if kind == "rays":
        return {"bytes": case["rays"] * 56.0, "flops": case["rays"] * RAY_FLOPS}
    if kind == "particles":
        return {"bytes": case["particles"] * (48 + 48 + 4.0), "flops": case["particles"] * 4 * RAY_FLOPS / 2}
    px = case["width"] * case["height"]
    if kind == "animated":
        inst = 201 + case["quads"]
        return {"bytes": 2 * (px * 16.0 + inst * 500.0 + 16e6),
                "flops": 2 * px * case["depth"] * RAYS_PER_PATH["field"] * RAY_FLOPS}
    if kind == "restir":
        rays = 6 + 1.5 * case["spatial"] + (3 if case["mode"] == "pt" else 0)
        return {"bytes": 2 * (px * (60.0 + 2 * 48) + 16e6), "flops": 2 * px * (rays * RAY_FLOPS + 64 * 150.0)}
    return {"bytes": px * 16.0 + 16e6 + 2 * 66304.0,
            "flops": (px + case["train_paths"]) * 6 * RAYS_PER_PATH["terrain"] * RAY_FLOPS
            + 0.25 * px * 33e3 + case["train_paths"] * 4 * 99e3}


def _views_only(case):
    """The sizes of a path case's views (no meshes made)."""
    w, h = case["width"], case["height"]
    if case["scene"] == "terrain" and case["views"] == 8:
        return [{"width": max(1, a * w // 3840), "height": max(1, b * h // 2160)}
                for a, b in scenes.CONFIG3_RESOLUTIONS]
    return [{"width": max(8, w >> (k % 3)), "height": max(8, h >> (k % 3))} for k in range(case["views"])]


# ---- the same in 64 bits ------------------------------------------------------------
def exact(case, seed):
    """TAA frames and small closest-hit queries; a frame's light paths or a large query against every triangle would
    take far longer than a few seconds in 64 bits."""
    if case["kind"] == "taa":
        return _exact_taa(prepare(case, seed)["frames"], case["width"], case["height"])
    if case["kind"] == "rays" and not case["any_hit"] and case["rays"] <= 256:
        return _exact_hits(_sphere_scene(seed), _rays(case, np.random.default_rng(seed)))
    return None


def _exact_hits(sc, rays):
    o = torch.from_numpy(rays["o"].astype(np.float64)).cuda()
    d = torch.from_numpy(rays["d"].astype(np.float64)).cuda()
    tmin = torch.from_numpy(rays["tmin"].astype(np.float64)).cuda()
    best = torch.from_numpy(rays["tmax"].astype(np.float64)).cuda()
    t_out, u_out, v_out = torch.full_like(best, -1.0), torch.zeros_like(best), torch.zeros_like(best)
    for inst in sc.instances:
        m = sc.meshes[int(inst["mesh_id"])]
        M = inst["transform"].reshape(3, 4).astype(np.float64)
        p = torch.from_numpy(m.positions.astype(np.float64) @ M[:, :3].T + M[:, 3]).cuda()
        ix = torch.from_numpy(m.indices.astype(np.int64)).cuda()
        for b in range(0, len(ix), 16384):
            a0, a1, a2 = (p[ix[b:b + 16384, k]] for k in range(3))
            e1, e2 = a1 - a0, a2 - a0
            h = torch.linalg.cross(d[:, None, :].expand(-1, len(e2), -1), e2[None].expand(len(d), -1, -1))
            det = (h * e1[None]).sum(-1)
            s = o[:, None, :] - a0[None]
            u = (s * h).sum(-1) / det
            q = torch.linalg.cross(s, e1[None].expand_as(s))
            v = (q * d[:, None, :]).sum(-1) / det
            t = (q * e2[None]).sum(-1) / det
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin[:, None]) & (det != 0)
            t = torch.where(ok, t, torch.full_like(t, math.inf))
            tm, k = t.min(1)
            row = torch.arange(len(d), device=d.device)
            near = tm < best
            best = torch.where(near, tm, best)
            t_out = torch.where(near, tm, t_out)
            u_out = torch.where(near, u[row, k], u_out)
            v_out = torch.where(near, v[row, k], v_out)
    return {"t": t_out, "u": u_out, "v": v_out, "inst": None, "prim": None, "flags": None}


def _exact_taa(frames, w, h):
    outs, hist, pmot = [], None, None
    for rad, mot in frames:
        cur, vel = rad.double().view(h, w, 4), mot.double().view(h, w, 2)
        hist = cur if hist is None else hist
        pmot = vel if pmot is None else pmot
        x = torch.arange(w, device=cur.device, dtype=torch.float64)[None, :].expand(h, w)
        y = torch.arange(h, device=cur.device, dtype=torch.float64)[:, None].expand(h, w)
        hx = ((x + 0.5) / w + vel[..., 0]).clamp(0.0, 1.0) * w - 0.5
        hy = ((y + 0.5) / h + vel[..., 1]).clamp(0.0, 1.0) * h - 0.5
        fx, fy = hx.floor(), hy.floor()
        a, b = (hx - fx)[..., None], (hy - fy)[..., None]
        i0, j0 = fx.long() % w, fy.long() % h
        i1, j1 = (fx.long() + 1) % w, (fy.long() + 1) % h

        def fetch(img):
            return (img[j0, i0] * ((1 - a) * (1 - b)) + img[j0, i1] * (a * (1 - b)) + img[j1, i0] * ((1 - a) * b)
                    + img[j1, i1] * (a * b))

        rows = torch.arange(-1, h + 1, device=cur.device).clamp(0, h - 1)
        cols = torch.arange(-1, w + 1, device=cur.device).clamp(0, w - 1)
        pad = cur[rows][:, cols][..., :3].clamp(min=0.0)
        nb = torch.stack([pad[dy:dy + h, dx:dx + w] for dx in range(3) for dy in range(3)])
        mu = nb.sum(0) / 9.0
        sigma = ((nb * nb).sum(0) / 9.0 - mu * mu).abs().sqrt()
        lo, hi = mu - 0.55 * sigma, mu + 0.55 * sigma
        p = torch.minimum(torch.maximum(mu, nb.amin(0)), nb.amax(0))
        r = fetch(hist)[..., :3].clamp(min=0.0) - p
        for c in range(3):
            top = hi[..., c] - p[..., c]
            r = torch.where((r[..., c] > top + 1e-8)[..., None], r * (top / r[..., c])[..., None], r)
        for c in range(3):
            low = lo[..., c] - p[..., c]
            r = torch.where((r[..., c] < low - 1e-8)[..., None], r * (low / r[..., c])[..., None], r)
        speed = (fetch(pmot) + vel).norm(dim=-1, keepdim=True)
        dis = ((speed - 0.001) * 10.0).clamp(0.0, 1.0)
        fin = (cur[..., :3] * 0.1 + (p + r) * 0.9) * (1 - dis) + mu * dis
        out = torch.cat([fin, torch.ones_like(fin[..., :1])], -1)
        outs.append(out.view(-1, 4))
        hist, pmot = out, vel
    return outs
