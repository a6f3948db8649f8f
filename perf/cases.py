"""The work a user of this framework has it do, as cases of one pass each through its public entry points.

Four kinds of call make up nearly all of it: ray queries (a picking tool's handful, a baking tool's
millions), renders (an editor's preview, a still, an animation frame whose geometry changed), batches
of small render jobs (a render service), and differentiable rendering (forward and backward in an
optimisation loop); light paths feed the bidirectional integrators.  The scenes are the repository's
own generators, made from the seed; sizes follow its benchmark and test configurations.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from seesharp_gb300 import FrameBuffer, PathTracer, _native, render_batch, workloads
from seesharp_gb300.adjoint import DifferentiableRender, l2_loss

SPHERE_TRIANGLES = 5120  # an icosphere of subdivision level 4, as the benchmark scenes have them


def listed():
    return [
        # a picking tool or an editor's gizmo: a few rays, where only latency counts
        {"name": "query_few", "kind": "query", "scene": "box", "spheres": 0, "rays": 97, "any": False, "device": False},
        # visibility between two sets of points (a light-baking or probe-placement pass), arrays on the host
        {"name": "occlusion_host", "kind": "query", "scene": "field", "spheres": 40, "rays": 65536, "any": True, "device": False},
        # closest hits of a million incoherent rays in the 1M-triangle scene, arrays on the device
        {"name": "query_million", "kind": "query", "scene": "field", "spheres": 200, "rays": 1000003, "any": False, "device": True},
        # an editor's interactive preview: one sample per pixel of a small window
        {"name": "preview", "kind": "render", "scene": "box", "spheres": 0, "width": 160, "height": 90, "spp": 1, "depth": 5, "shadow": 1, "variance": False},
        # the small benchmark configuration: a diffuse Cornell box, 256 x 256, 16 samples, depth 5
        {"name": "still_box", "kind": "render", "scene": "box", "spheres": 0, "width": 256, "height": 256, "spp": 16, "depth": 5, "shadow": 1, "variance": False},
        # textured and rough materials at an odd resolution, with two shadow rays per vertex and the variance layer
        {"name": "still_materials", "kind": "render", "scene": "materials", "spheres": 0, "width": 509, "height": 383, "spp": 32, "depth": 6, "shadow": 2,
         "variance": True},
        # the headline benchmark configuration: the 1M-triangle scene, 1024 x 1024, 64 samples, depth 8
        {"name": "still_field", "kind": "render", "scene": "field", "spheres": 200, "width": 1024, "height": 1024, "spp": 64, "depth": 8, "shadow": 1,
         "variance": False},
        # an animation frame: the geometry changed, so the scene is prepared again (upload, BVH) and rendered at a few samples
        {"name": "frame", "kind": "frame", "scene": "field", "spheres": 120, "width": 960, "height": 540, "spp": 2, "depth": 6, "shadow": 1, "variance": False},
        # a render service: uneven small jobs in one batch (64^2 to 256^2 pixels, 1 to 16 samples, 10k to 200k triangles)
        {"name": "batch", "kind": "batch", "jobs": 40},
        # an optimisation step on the differentiation configuration: 512 x 512, 32 samples, depth 5, a 256^2 texture
        {"name": "gradient_box", "kind": "gradient", "scene": "materials", "spheres": 0, "quads": 0, "texture": 256, "width": 512, "height": 512, "spp": 32,
         "depth": 5, "views": 0},
        # the same on a slice of the large combined job: a textured terrain, many rough spheres, several camera views in one batch
        {"name": "gradient_views", "kind": "gradient", "scene": "terrain", "spheres": 300, "quads": 512, "texture": 512, "width": 640, "height": 360, "spp": 8,
         "depth": 10, "views": 3},
        # light subpaths for a bidirectional integrator
        {"name": "light_paths", "kind": "light", "scene": "field", "spheres": 60, "rays": 100000, "depth": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "render", "render", "render", "frame", "batch", "gradient", "gradient", "light"])
    if kind == "query":
        scene = rng.choice(["box", "field", "field"])
        return {"kind": kind, "scene": scene, "spheres": _log(rng, 2, 200) if scene == "field" else 0, "rays": _log(rng, 16, 2000000),
                "any": rng.random() < 0.5, "device": rng.random() < 0.5}
    if kind == "light":
        return {"kind": kind, "scene": "field", "spheres": _log(rng, 2, 120), "rays": _log(rng, 1000, 150000), "depth": rng.randint(2, 8)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(6, 40)}
    if kind == "gradient":
        w, h = _log(rng, 64, 640), _log(rng, 64, 512)
        spp = min(_log(rng, 2, 32), max(1, 8000000 // (w * h)))
        if rng.random() < 0.6:
            return {"kind": kind, "scene": "materials", "spheres": 0, "quads": 0, "texture": _log(rng, 16, 512), "width": w, "height": h, "spp": spp,
                    "depth": rng.randint(2, 8), "views": 0}
        return {"kind": kind, "scene": "terrain", "spheres": _log(rng, 10, 300), "quads": _log(rng, 32, 512), "texture": _log(rng, 16, 512), "width": w,
                "height": h, "spp": min(spp, 8), "depth": rng.randint(3, 10), "views": rng.randint(1, 3)}
    w, h = _log(rng, 48, 1920), _log(rng, 48, 1080)
    if kind == "frame":
        return {"kind": kind, "scene": "field", "spheres": _log(rng, 4, 200), "width": w, "height": h, "spp": rng.randint(1, 4), "depth": rng.randint(2, 8),
                "shadow": 1, "variance": False}
    spp = min(_log(rng, 1, 64), max(1, 30000000 // (w * h)))
    scene = rng.choice(["box", "materials", "field", "field", "sky"])
    return {"kind": kind, "scene": scene, "spheres": _log(rng, 2, 200) if scene == "field" else 0, "width": w, "height": h, "spp": spp,
            "depth": rng.randint(2, 8), "shadow": rng.choice([1, 1, 1, 2]), "variance": rng.random() < 0.25}


def _scene(case, seed, width, height):
    if case["scene"] == "box":
        return workloads.cornell_box(width, height, seed=seed)
    if case["scene"] == "materials":
        rough = np.random.default_rng(seed).uniform(0.15, 0.8, 2)
        return workloads.cornell_box_differentiable(width, height, seed=seed, roughness=(float(rough[0]), float(rough[1])))[0]
    if case["scene"] == "sky":
        return workloads.env_lit_box(width, height, seed=seed)
    return workloads.sphere_field(case["spheres"], width, height, seed=seed)


def _rays(case, seed):
    """Rays between points of the scene's volume: closest-hit rays along uniform directions, occlusion
    rays as segments (tmax just below one, as IsOccluded traces them)."""
    g = torch.Generator().manual_seed(seed)
    n = case["rays"]
    lo, hi = (-0.95, 0.95) if case["scene"] == "box" else (0.0, 20.0)
    a = torch.rand((n, 3), generator=g) * (hi - lo) + lo
    b = torch.rand((n, 3), generator=g) * (hi - lo) + lo
    if not case["any"]:
        d = torch.randn((n, 3), generator=g)
        b = a + d / d.norm(dim=1, keepdim=True)
    rays = torch.zeros((n, 8))
    rays[:, 0:3] = a
    rays[:, 4:7] = b - a
    rays[:, 7] = 1.0 - 1e-5 if case["any"] else math.inf
    return rays


def _integrator(case, seed):
    return PathTracer(TotalSpp=case["spp"], MaxDepth=case["depth"], BaseSeed=0xC030114 + seed, NumShadowRays=case.get("shadow", 1))


def _film(case):
    flags = FrameBuffer.Flags.Recommended
    if case.get("variance"):
        flags |= FrameBuffer.Flags.EstimatePixelVariance
    return FrameBuffer(case["width"], case["height"], flags=flags)


def _batch_jobs(case, seed):
    """Uneven serving jobs: the mix of resolutions, samples, depths and triangle counts belongs to the
    case, the scenes and the base seeds to the seed."""
    mix, rng = np.random.default_rng(case["jobs"]), np.random.default_rng(seed)
    out = []
    for k in range(case["jobs"]):
        size, spp, depth = int(mix.choice([64, 128, 256])), int(mix.integers(1, 17)), int(mix.integers(3, 9))
        spheres = max(1, int(round(math.exp(mix.uniform(math.log(1e4), math.log(2e5))) / SPHERE_TRIANGLES)))
        sc = workloads.sphere_field(spheres, size, size, seed=int(rng.integers(1 << 30)))
        out.append((sc, PathTracer(TotalSpp=spp, MaxDepth=depth, BaseSeed=int(rng.integers(1 << 31)))))
    return out


def prepare(case, seed):
    case = dict(case)
    kind = case["kind"]
    state = {"case": case, "kind": kind}
    if kind == "query":
        sc = _scene(case, seed, 64, 64)
        sc.Prepare()
        rays = _rays(case, seed)
        state.update(scene=sc, rays=rays.cuda() if case["device"] else rays.numpy())
    elif kind in ("render", "frame"):
        sc = _scene(case, seed, case["width"], case["height"])
        if kind == "render":
            sc.Prepare()
        state.update(scene=sc, integrator=_integrator(case, seed))
    elif kind == "light":
        sc = _scene(case, seed, 64, 64)
        sc.Prepare()
        state.update(scene=sc, seed=0x5EED + seed)
    elif kind == "batch":
        jobs = _batch_jobs(case, seed)
        for sc, _ in jobs:
            sc.Prepare()
        state.update(jobs=jobs)
    else:
        rng = np.random.default_rng(seed)
        w, h = case["width"], case["height"]
        if case["scene"] == "materials":
            sc, tex, mats, lights = workloads.cornell_box_differentiable(w, h, seed=seed, tex_res=case["texture"])
            groups, views = [lights], None
        else:
            sc, tex, mats, views = workloads.large_combined(w, h, seed=seed, num_spheres=case["spheres"], terrain_quads=case["quads"], tex_res=case["texture"],
                                                            num_lights=100, views=max(1, case["views"]))
            groups = []
        sc.Prepare()
        dr = DifferentiableRender(sc, _integrator(case, seed), texture=tex, roughness_materials=mats, emitters=groups, views=views)
        yy, xx = np.meshgrid(np.linspace(0, 1, h), np.linspace(0, 1, w), indexing="ij")
        f = rng.uniform(2, 9, 3)
        target = np.stack([0.3 + 0.2 * np.sin(f[k] * xx) * np.cos(f[k] * yy) for k in range(3)], -1).astype(np.float32)
        # the parameters of this optimisation step, slightly off the scene's own
        state.update(scene=sc, dr=dr, target=target, texture=np.clip(tex.Image.data * rng.uniform(0.9, 1.1), 0.02, 0.98).astype(np.float32),
                     roughness=rng.uniform(0.2, 0.8, len(mats)).astype(np.float32),
                     radiance=rng.uniform(4, 17, (1, 3)).astype(np.float32) if groups else None)
    return state


def _hits(raw):
    """A query's hit records (SstHit: distance, u, v, ids, error offset, position, normal) by type."""
    if isinstance(raw, torch.Tensor):
        ids = raw[:, 3:5].contiguous().view(torch.int32)
    else:
        ids = np.ascontiguousarray(raw[:, 3:5]).view(np.int32)
    return {"duv": raw[:, 0:3], "ids": ids, "surface": raw[:, 5:12]}


def _render(state):
    sc, case = state["scene"], state["case"]
    fb = sc.FrameBuffer
    state["integrator"].Render(sc)
    out = {"film": fb.Image.data, "albedo": fb.layers["albedo"].Image.data, "normal": fb.layers["normal"].Image.data,
           "outliers": fb.OutlierCache.weight, "outlier_iterations": fb.OutlierCache.iteration}
    if case.get("variance"):
        out["variance"] = fb.PixelVariance.Image.data
    return out


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "query":
        sh = state["scene"].native
        rays = state["rays"]
        if not case["device"]:
            return {"occluded": sh.occluded(rays)} if case["any"] else _hits(sh.trace(rays))
        # the C ABI on device arrays, as a native host calls it
        n = rays.shape[0]
        p = ctypes.c_void_p(rays.data_ptr())
        if case["any"]:
            occ = torch.empty(n, dtype=torch.int32, device="cuda")
            _native.check(sh.lib.sst_occluded(sh.handle, p, n, ctypes.c_void_p(occ.data_ptr()), _native.SST_MEM_DEVICE))
            return {"occluded": occ}
        hits = torch.empty((n, 12), device="cuda")
        _native.check(sh.lib.sst_trace(sh.handle, p, n, ctypes.c_void_p(hits.data_ptr()), _native.SST_MEM_DEVICE))
        return _hits(hits)
    if kind in ("render", "frame"):
        state["scene"].FrameBuffer = _film(case)
        if kind == "frame":
            state["scene"].Prepare()
        return _render(state)
    if kind == "light":
        floats, ints, lengths, _ = state["scene"].native.trace_light_paths(state["seed"], 0, case["rays"], case["depth"])
        return {"vertices": floats, "ids": ints, "lengths": lengths}
    if kind == "batch":
        for sc, _ in state["jobs"]:
            sc.FrameBuffer = FrameBuffer(sc.FrameBuffer.Width, sc.FrameBuffer.Height)
        render_batch(state["jobs"])
        return [sc.FrameBuffer.Image.data for sc, _ in state["jobs"]]
    dr = state["dr"]
    image = dr.forward(state["texture"], state["roughness"], state["radiance"])
    if isinstance(image, list):
        grad = dr.backward([l2_loss(i, state["target"])[1] for i in image])
    else:
        grad = dr.backward(l2_loss(image, state["target"])[1])
    return {"image": image, "texture": grad["texture"], "roughness": grad["roughness"], "radiance": grad["radiance"],
            "base": grad["raw"]["materialBaseColor"], "emitters": grad["raw"]["emitterRadiance"]}


def _triangles(case):
    if case["kind"] == "batch":
        return int(case["jobs"] * 6.3e4)
    if case["scene"] == "terrain":
        return case["spheres"] * SPHERE_TRIANGLES + 2 * case["quads"] ** 2 + 100
    return {"box": 36, "materials": 36, "sky": 14}.get(case["scene"]) or case["spheres"] * SPHERE_TRIANGLES + 52


def work(case):
    """Bytes: what comes in and goes out, and the scene (48 bytes of positions per triangle, 48 of
    shading records where it is shaded) once.  Operations: per ray two boxes per level of a balanced
    binary tree (24 operations a box) and one triangle (60); per shaded vertex 400."""
    tris = _triangles(case)
    ray = 48.0 * math.ceil(math.log2(max(2, tris))) + 60.0
    kind = case["kind"]
    if kind == "query":
        n = case["rays"]
        return {"bytes": n * (36.0 if case["any"] else 80.0) + 48.0 * tris, "flops": n * ray}
    if kind == "light":
        n = case["rays"]
        return {"bytes": n * (case["depth"] + 1) * 88.0 + 96.0 * tris, "flops": n * min(3.0, case["depth"]) * (ray + 400.0)}
    if kind == "batch":
        samples, pixels = case["jobs"] * 2.4e5, case["jobs"] * 2.9e4
        return {"bytes": pixels * 12.0 + 96.0 * tris, "flops": samples * 2.8 * (2.3 * ray + 400.0)}
    samples = float(case["width"] * case["height"] * case["spp"] * max(1, case.get("views", 1)))
    # vertices of a path: open scenes lose about a third of the rays per bounce, Russian roulette starts at depth 5
    per = min(case["depth"], 4.5) if case["scene"] in ("box", "materials") else min(case["depth"], 2.8)
    flops = samples * per * (ray * (1 + case.get("shadow", 1)) + 400.0 * (1 + case.get("shadow", 1)))
    pixels = float(case["width"] * case["height"] * max(1, case.get("views", 1)))
    if kind == "gradient":
        return {"bytes": pixels * 24.0 + samples * 24.0 + 96.0 * tris + 24.0 * case["texture"] ** 2, "flops": 2.5 * flops}
    return {"bytes": pixels * (12 + 24 + 32 + (12 if case["variance"] else 0)) + 96.0 * tris, "flops": flops}


def exact(case, seed):
    """The closest hits in 64 bits: every ray against the triangles of each mesh whose bounding sphere
    it meets.  Renders, light paths and gradients follow 32-bit random decisions and have no such value;
    occlusion flags are whole numbers."""
    if case["kind"] != "query" or case["any"] or case["rays"] > 1100000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sc = _scene(case, seed, 64, 64)
    rays = _rays(case, seed).to(dev).double()
    o, d = rays[:, 0:3], rays[:, 4:7]
    n = rays.shape[0]
    best = torch.full((n,), math.inf, dtype=torch.float64, device=dev)
    u = torch.zeros(n, dtype=torch.float64, device=dev)
    v = torch.zeros_like(u)
    surface = torch.zeros((n, 7), dtype=torch.float64, device=dev)
    step = 1 << 24
    for mesh in sc.Meshes:
        tri = torch.from_numpy(mesh.Vertices[mesh.Indices.reshape(-1, 3)]).to(dev).double()
        v1, v2, v3 = tri[:, 0], tri[:, 1], tri[:, 2]
        e1, e2 = v2 - v1, v3 - v1
        normal = torch.linalg.cross(e1, e2)
        centre = tri.reshape(-1, 3).mean(0)
        radius = (tri.reshape(-1, 3) - centre).norm(dim=1).max() * 1.001
        oc = centre - o
        along = (oc * d).sum(1) / (d * d).sum(1)
        off = (oc - along[:, None] * d).norm(dim=1)
        idx = torch.nonzero((off <= radius) & ((along > 0) | (oc.norm(dim=1) <= radius))).squeeze(1)
        rows = max(1, step // tri.shape[0])
        for at in range(0, idx.numel(), rows):
            i = idx[at:at + rows]
            ro, rd = o[i][:, None, :], d[i][:, None, :]
            # Cramer's rule on o + t d = v1 + u e1 + v e2
            det = -(rd * normal).sum(2)
            s = ro - v1
            t = (s * normal).sum(2) / det
            q = torch.linalg.cross(s, rd.expand_as(s), dim=2)
            uu = (e2 * q).sum(2) / det
            vv = -(e1 * q).sum(2) / det
            t = torch.where((uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (t > 0), t, math.inf)
            tm, k = t.min(1)
            hit = tm < best[i]
            j, k, r = i[hit], k[hit], torch.arange(i.numel(), device=dev)[hit]
            best[j] = tm[hit]
            u[j], v[j] = uu[r, k], vv[r, k]
            w = 1 - u[j] - v[j]
            a, b, c = u[j][:, None] * v2[k], v[j][:, None] * v3[k], w[:, None] * v1[k]
            surface[j, 0] = (a.abs() + b.abs() + c.abs()).norm(dim=1) * 32 * 1.19209e-07
            surface[j, 1:4] = a + b + c
            surface[j, 4:7] = normal[k] / normal[k].norm(dim=1, keepdim=True)
    best = torch.where(torch.isinf(best), torch.zeros_like(best), best)
    return {"duv": torch.stack([best, u, v], 1), "ids": None, "surface": surface}
