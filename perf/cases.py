"""Performance cases: what a user of the framework has it do.

Whole images (``PTRenderer.Render``), batches of images
(``Context.render_batch``), photon-mapped images (``SPPMRenderer.Render``),
ray queries (``GpuScene.Intersect`` / ``Occlude``) and loading a scene
(``GpuScene``: upload and tree build) up to its first image or pick, from the
smallest call to the benchmark's scene of 1.3 million triangles.

``listed()`` holds the fixed cases and ``draw(rng)`` gives more of the same
ranges.  ``prepare(case, seed)`` makes the inputs a program has in hand,
``run(state)`` is one pass through the public interface, ``work(case)`` a
lower bound of its bytes and operations, and ``exact(case, seed)`` the
float64 answer where a brute-force one is affordable.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ajisai_render_gb300 import api, scenes

F32 = np.float32


def listed():
    return [
        # the smallest call: one sample per pixel of a small box, as an
        # interactive viewer asks for on every camera move
        dict(name="box_preview", kind="frame", scene="box", size=0, width=128,
             height=128, spp=1, min_bounces=3, max_bounces=8, mis=True,
             fp64=False, drop=False, tri_test=0),
        # the Cornell-style configuration at its own size
        dict(name="box_frame", kind="frame", scene="box", size=0, width=256,
             height=256, spp=64, min_bounces=3, max_bounces=8, mis=True,
             fp64=False, drop=False, tri_test=0),
        # mirror, glass, metal, plastic and an area light at an odd size, as a
        # ground-truth render: float64 film, non-finite samples left out
        dict(name="materials_frame", kind="frame", scene="materials", size=0,
             width=311, height=233, spp=24, min_bounces=5, max_bounces=10,
             mis=True, fp64=True, drop=True, tri_test=0),
        # the single-job benchmark's scene, film and depth at fewer samples
        dict(name="sphere_frame", kind="frame", scene="sphere", size=8,
             width=1024, height=1024, spp=32, min_bounces=5, max_bounces=16,
             mis=True, fp64=False, drop=False, tri_test=0),
        # random-box clutter without MIS (the reference's use_mis: false) and
        # with the watertight test, on a film of no round size
        dict(name="clutter_frame", kind="frame", scene="clutter", size=9001,
             width=853, height=479, spp=16, min_bounces=5, max_bounces=10,
             mis=False, fp64=False, drop=False, tri_test=1),
        # small images of several scenes in one call (a thumbnail service)
        dict(name="batch_small", kind="batch", jobs=16, size=5, low=64,
             high=256, spp=24, max_bounces=12),
        # photon mapping with the reference's defaults for everything but the
        # iteration count
        dict(name="sppm_box", kind="sppm", scene="area", size=0, width=192,
             height=192, iterations=12, photons=100000, radius=0.1,
             camera_depth=8),
        # photon mapping at the benchmark's film size, photon count and radius
        dict(name="sppm_sphere", kind="sppm", scene="sphere", size=7,
             width=512, height=512, iterations=4, photons=2000000, radius=0.01,
             camera_depth=8),
        # closest hits of a few thousand rays (picking, probes)
        dict(name="pick_rays", kind="rays", scene="clutter", size=401,
             rays=4999, query="closest", tri_test=0),
        # visibility of millions of point pairs (ambient occlusion baking)
        dict(name="visibility_rays", kind="rays", scene="sphere", size=7,
             rays=2000003, query="any", tri_test=0),
        # opening a small scene: tree build up to the first picked objects
        dict(name="load_clutter", kind="load", scene="clutter", size=851,
             width=0, height=0, rays=1021, tri_test=0),
        # opening the benchmark's scene: upload, tree build and a first image
        dict(name="load_sphere", kind="load", scene="sphere", size=8,
             width=640, height=360, rays=0, tri_test=0),
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene_size(rng, scene):
    if scene == "sphere":
        return rng.randint(3, 8)
    return _log(rng, 50, 20000) if scene == "clutter" else 0


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "sppm", "rays", "rays", "load"])
    scene = rng.choice(["box", "area", "materials", "sphere", "sphere", "clutter"])
    if kind == "frame":
        width, height = _log(rng, 32, 1100), _log(rng, 32, 1100)
        most = 20e6 if scene in ("box", "sphere") else 5e6
        spp = _log(rng, 1, max(1, min(128, int(most / (width * height)))))
        return dict(kind=kind, scene=scene, size=_scene_size(rng, scene), width=width,
                    height=height, spp=spp, min_bounces=rng.choice([3, 5]),
                    max_bounces=rng.choice([4, 8, 10, 12, 16]), mis=rng.random() < 0.8,
                    fp64=rng.random() < 0.2, drop=rng.random() < 0.2,
                    tri_test=1 if rng.random() < 0.2 else 0)
    if kind == "batch":
        high = rng.choice([128, 256, 384])
        return dict(kind=kind, jobs=rng.randint(2, 24), size=rng.randint(3, 6),
                    low=rng.choice([32, 64, 100]), high=high, spp=_log(rng, 1, 32),
                    max_bounces=rng.choice([8, 12]))
    if kind == "sppm":
        # the boxes are a unit across, the other scenes four and more
        box = scene in ("box", "area", "materials")
        most = 192 if box else 512
        return dict(kind=kind, scene=scene, size=min(_scene_size(rng, scene), 4000),
                    width=_log(rng, 48, most), height=_log(rng, 48, most),
                    iterations=rng.randint(1, 8),
                    photons=_log(rng, 20000, 150000 if box else 1000000),
                    radius=rng.choice([0.02, 0.1] if box else [0.01, 0.02]),
                    camera_depth=rng.choice([4, 8]))
    if kind == "rays":
        return dict(kind=kind, scene=scene, size=_scene_size(rng, scene),
                    rays=_log(rng, 1, 2000003), query=rng.choice(["closest", "any"]),
                    tri_test=1 if rng.random() < 0.2 else 0)
    frame = rng.random() < 0.5
    return dict(kind=kind, scene=scene, size=_scene_size(rng, scene),
                width=_log(rng, 32, 320) if frame else 0,
                height=_log(rng, 32, 320) if frame else 0,
                rays=0 if frame else _log(rng, 1, 5000), tri_test=0)


# ------------------------------------------------------------------ scenes --
_DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=None)
def _sphere_topology(subdiv):
    """The icosphere before it is displaced: the same for every seed."""
    v, f = scenes.icosphere(subdiv)
    return torch.from_numpy(v).to(_DEVICE), np.ascontiguousarray(f, np.int32)


def _displaced_sphere(subdiv, rng, waves=24):
    """The icosphere displaced radially by about 0.15 of its radius: a seeded
    sum of plane waves from 2 to 32 periods, with the surface's normals."""
    v, f = _sphere_topology(subdiv)
    freq = 2.0 * np.exp2(rng.uniform(0.0, 4.0, waves))
    k = rng.normal(size=(waves, 3))
    k *= (freq / np.linalg.norm(k, axis=1))[:, None]
    phase = rng.uniform(0.0, 2 * np.pi, waves)
    amp = 0.15 / freq * 2.0 / math.sqrt(waves / 4)
    r = torch.ones_like(v[:, 0])
    g = torch.zeros_like(v)
    for i in range(waves):
        arg = v[:, 0] * k[i, 0] + v[:, 1] * k[i, 1] + v[:, 2] * k[i, 2] + phase[i]
        r += amp[i] * torch.sin(arg)
        c = amp[i] * torch.cos(arg)
        for a in range(3):
            g[:, a] += c * k[i, a]
    along = g[:, 0] * v[:, 0] + g[:, 1] * v[:, 1] + g[:, 2] * v[:, 2]
    n = r[:, None] * v - (g - along[:, None] * v)
    n = n / torch.sqrt(n[:, 0] ** 2 + n[:, 1] ** 2 + n[:, 2] ** 2)[:, None]
    return ((r[:, None] * v).float().cpu().numpy(), n.float().cpu().numpy(), f)


def _camera(rng, width, height, dist, target):
    """A pinhole camera on a seeded sphere around the scene."""
    az = rng.uniform(0.0, 2 * math.pi)
    el = math.radians(rng.uniform(5.0, 45.0))
    pos = [target[0] + dist * math.cos(el) * math.sin(az),
           target[1] + dist * math.sin(el),
           target[2] + dist * math.cos(el) * math.cos(az)]
    return scenes.Camera(tuple(pos), tuple(target), (0.0, 1.0, 0.0), 40.0, width, height)


def _scene(name, size, rng, width, height):
    """The flat scene and its camera record."""
    width, height = max(1, width), max(1, height)
    if name in ("box", "area", "materials"):
        make = {"box": scenes.cornell_box, "area": scenes.cornell_area,
                "materials": scenes.material_box}[name]
        sc = make(width, height)
        x, y = rng.uniform(-0.1, 0.1, 2)
        sc.camera.position = (float(x), float(y), 1.9)
    else:
        if name == "sphere":
            pos, nrm, idx = _displaced_sphere(size, rng)
            mats = [scenes.disney_params(rng)]
            prims = [scenes.Mesh(pos, idx, nrm, 0, False)]
        else:
            mats, prims = [], []
            for k, (p, idx) in enumerate(scenes.clutter_meshes(size, rng, 16)):
                mats.append(scenes.disney_params(rng))
                prims.append(scenes.Mesh(p, idx, None, k, False))
        mats.append(scenes.Diffuse((0.5, 0.5, 0.5)))
        s, y = 8.0, -1.2
        prims.append(scenes.Quad((-s, y, s), (s, y, s), (s, y, -s), (-s, y, -s),
                                 len(mats) - 1, True))
        lights = [scenes.DirectionalLight((0.3, 1.0, 0.2), 2.0), scenes.EnvLight(0.5)]
        sc = scenes.Scene(prims, mats, lights,
                          _camera(rng, width, height, 3.6, (0.0, -0.1, 0.0)))
    flat = scenes.flatten(sc)
    return flat, flat.camera


def _rays(name, n, rng, query):
    """Rays into the scene: origins around it aimed at points inside, with a
    finite reach for visibility queries."""
    near, far = (0.4, 1.5) if name in ("box", "area", "materials") else (1.0, 2.5)
    o = rng.uniform(-far, far, (n, 3))
    at = rng.uniform(-near, near, (n, 3))
    d = at - o
    length = np.linalg.norm(d, axis=1, keepdims=True)
    d /= np.maximum(length, 1e-9)
    tmax = length if query == "any" else np.full((n, 1), np.inf)
    return np.concatenate([o, d, np.full((n, 1), 1e-4), tmax], 1).astype(F32)


@functools.lru_cache(maxsize=None)
def _context():
    """One context per process, as a program keeps it."""
    return api.Context(0)


def _gpu_scene(flat, tri_test=0):
    return api.CreateDefaultScene(_context(), flat, api.CreatePLOCAggregate(16, tri_test))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "batch":
        ctx = _context()
        made = []
        for name, size in (("sphere", case["size"]), ("clutter", 400 * case["size"]),
                           ("box", 0), ("area", 0)):
            flat, _ = _scene(name, size, rng, 8, 8)
            made.append((name, _gpu_scene(flat)))
        jobs = []
        sizes = np.random.default_rng(case["jobs"] + case["high"])  # not of the seed
        for i in range(case["jobs"]):
            name, scene = made[i % len(made)]
            w, h = (int(x) for x in sizes.integers(case["low"], case["high"] + 1, 2))
            spp = int(sizes.integers(max(1, case["spp"] // 2), case["spp"] * 2 + 1))
            if name in ("box", "area"):
                cam = scenes.Camera((0.0, 0.0, 1.9), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0),
                                    40.0, w, h)
            else:
                cam = _camera(rng, w, h, 3.6, (0.0, -0.1, 0.0))
            args = api.PTRendererArgs(spp=spp, max_bounces=case["max_bounces"])
            jobs.append((scene, cam.pack(), api.CreatePTRenderer(args, seed=seed + i)))
        return dict(kind=kind, ctx=ctx, jobs=jobs, scenes=made)
    flat, cam = _scene(case["scene"], case["size"], rng, case.get("width", 0),
                       case.get("height", 0))
    if kind == "load":
        args = api.PTRendererArgs(spp=1, max_bounces=4)
        return dict(kind=kind, flat=flat, camera=cam, frame=case["width"] > 0,
                    renderer=api.CreatePTRenderer(args, seed=seed),
                    rays=_rays(case["scene"], case["rays"], rng, "closest"))
    scene = _gpu_scene(flat, case.get("tri_test", 0))
    if kind == "frame":
        args = api.PTRendererArgs(spp=case["spp"], min_bounces=case["min_bounces"],
                                  max_bounces=case["max_bounces"], use_mis=case["mis"])
        return dict(kind=kind, scene=scene, camera=cam,
                    renderer=api.PTRenderer(args, seed, case["fp64"], case["drop"]))
    if kind == "sppm":
        args = api.SPPMRendererArgs(forward_max_depth=case["camera_depth"],
                                    init_radius=case["radius"],
                                    iteration_count=case["iterations"],
                                    photons_per_iteration=case["photons"])
        return dict(kind=kind, scene=scene, camera=cam,
                    renderer=api.CreateSPPMRenderer(args, seed=seed))
    return dict(kind=kind, scene=scene, query=case["query"],
                rays=_rays(case["scene"], case["rays"], rng, case["query"]))


# --------------------------------------------------------------------- run --
def run(state):
    kind = state["kind"]
    if kind in ("frame", "sppm"):
        return state["renderer"].Render(state["scene"], state["camera"]).rgbw
    if kind == "batch":
        return [film.rgbw for film, _ in state["ctx"].render_batch(state["jobs"])]
    if kind == "rays":
        if state["query"] == "any":
            return state["scene"].Occlude(state["rays"])
        return state["scene"].Intersect(state["rays"])
    scene = _gpu_scene(state["flat"])
    if state["frame"]:
        out = state["renderer"].Render(scene, state["camera"]).rgbw
    else:
        out = scene.Intersect(state["rays"])
    scene.release()
    return out


# -------------------------------------------------------------------- work --
def _triangles(scene, size):
    if scene == "sphere":
        return 20 * 4 ** size + 2
    if scene == "clutter":
        return 12 * size + 2
    return {"box": 34, "area": 130, "materials": 356}[scene]


def _ray_flops(n):
    """One ray: a box test (18 operations) per level of a binary tree of n
    leaves and one triangle test (46)."""
    return 18 * max(1.0, math.log2(n)) + 46


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = [_triangles("sphere", case["size"]), _triangles("clutter", 400 * case["size"]),
             _triangles("box", 0), _triangles("area", 0)]
        side = 0.5 * (case["low"] + case["high"])
        px = case["jobs"] * side * side
        return {"bytes": sum(n) * 36 + 16 * px,
                "flops": 1.25 * case["spp"] * px * _ray_flops(sum(n) / 4)}
    n = _triangles(case["scene"], case["size"])
    px = case.get("width", 0) * case.get("height", 0)
    if kind == "frame":
        # every sample traces at least its camera ray
        return {"bytes": 36 * n + 16 * px, "flops": case["spp"] * px * _ray_flops(n)}
    if kind == "sppm":
        rays = px + case["iterations"] * case["photons"]
        return {"bytes": 36 * n + 16 * px, "flops": rays * _ray_flops(n)}
    if kind == "rays":
        out = 16 if case["query"] == "closest" else 1
        return {"bytes": 36 * n + case["rays"] * (32 + out), "flops": case["rays"] * _ray_flops(n)}
    # vertices, normals, material and flags in; a tree of 2n-1 boxes made
    return {"bytes": n * (36 + 36 + 8) + 2 * n * 32 + 16 * px + 48 * case["rays"],
            "flops": (px + case["rays"]) * _ray_flops(n) + 18 * 2 * n}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Closest hits by testing every triangle in float64 (Moller-Trumbore,
    the lowest index winning a tie); the other cases' answers are whole
    stochastic renders."""
    if case["kind"] not in ("rays", "load") or not case["rays"]:
        return None
    if case.get("query", "closest") != "closest":
        return None
    n = _triangles(case["scene"], case["size"])
    if case["rays"] * n > 2_000_000_000:
        return None
    rng = np.random.default_rng([seed, 77])
    flat, _ = _scene(case["scene"], case["size"], rng, case.get("width", 0),
                     case.get("height", 0))
    rays = torch.from_numpy(_rays(case["scene"], case["rays"], rng, "closest")).to(_DEVICE).double()
    tri = torch.from_numpy(flat.tris).to(_DEVICE).double().reshape(-1, 3, 3)
    v0, e0, e1 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]

    def cross(a, b):
        return torch.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1],
                            a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                            a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)

    ts, us, vs = [], [], []
    step = max(1, 20_000_000 // n)
    for k in range(0, rays.shape[0], step):
        r = rays[k:k + step]
        o, d = r[:, None, 0:3], r[:, None, 3:6]
        h = cross(d, e1[None])
        a = (e0[None] * h).sum(-1)
        s = o - v0[None]
        q = cross(s, e0[None].expand_as(s))
        u = (s * h).sum(-1) / a
        v = (d * q).sum(-1) / a
        t = (e1[None] * q).sum(-1) / a
        hit = ((a.abs() >= 1e-6) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
               & (t > r[:, 6:7]) & (t < r[:, 7:8]))
        t = torch.where(hit, t, torch.full_like(t, math.inf))
        best, i = t.min(1)
        found = torch.isfinite(best)
        ts.append(best)
        us.append(torch.where(found, u.gather(1, i[:, None])[:, 0], torch.zeros_like(best)))
        vs.append(torch.where(found, v.gather(1, i[:, None])[:, 0], torch.zeros_like(best)))
    return [torch.cat(ts).cpu().numpy(), None, torch.cat(us).cpu().numpy(),
            torch.cat(vs).cpu().numpy()]
