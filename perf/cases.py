"""The calls whose speed matters to a user of the renderer, over the sizes they are made at.

Every case goes through a public entry point of `snogray_b200`: ray queries
(`Scene.trace_device`, `Scene.trace`), one job on the plain renderer
(`Scene.render_device`, `Scene.render_window`), one or many jobs on the
streaming engine (`Engine.render`), and a scene's creation with its first
query.  `listed()` names them; `draw(rng)` gives more of the same ranges.

A case is a dict of plain values:
  call     "trace" | "trace_host" | "render" | "window" | "frame" | "jobs" | "load"
  scene    which generator of snogray_b200.scenes ("soup", "mixed", "terrain",
           "cornell", "mirror", "spot_far", "nested_glass", "mesh_smooth",
           "mesh_flat"); n: its size (triangles, or the terrain's grid side)
  rays, closest, normals                  for ray queries
  width, height, spp, depth, direct       for renders (direct: light samples of
                                          the direct-lighting integrator, 0 for
                                          the path integrator)
  n (most triangles of a job), jobs       for "jobs"
"""

from __future__ import annotations

import math

import numpy as np
import torch

import snogray_b200 as sb
from snogray_b200 import scenes

# Scenes with a fixed geometry (the terrain too): a seed changes the camera and
# the samples.  Random glass spheres may overlap five deep, which a render
# refuses.
_FIXED = {"cornell": scenes.cornell_box, "mirror": scenes.mirror_scene, "spot_far": scenes.spot_far_scene,
          "nested_glass": scenes.nested_glass_scene, "mesh_smooth": lambda: scenes.mesh_scene(True),
          "mesh_flat": lambda: scenes.mesh_scene(False)}


def _trace(name, scene, n, rays, closest, normals=False, call="trace"):
    return {"name": name, "call": call, "scene": scene, "n": n, "rays": rays, "closest": closest,
            "normals": normals}


def _render(name, call, scene, n, width, height, spp, depth, direct=0):
    return {"name": name, "call": call, "scene": scene, "n": n, "width": width, "height": height, "spp": spp,
            "depth": depth, "direct": direct}


def listed():
    return [
        # A picking or visibility query of an interactive tool: few rays, latency counts.
        _trace("trace_few", "soup", 10_000, 999, 999),
        # A baker's batch over all three primitive kinds, with normals, an odd count.
        _trace("trace_mixed", "mixed", 20_000, 1_000_003, 700_001, normals=True),
        # The intersection benchmark: 1M random triangles, 16M rays, half closest, half any-hit.
        _trace("trace_16m", "soup", 1 << 20, 1 << 24, 1 << 23),
        # A CPU program that sends its rays from host memory and reads hits, normals and counts back.
        _trace("trace_host", "terrain", 256, 300_001, 200_000, normals=True, call="trace_host"),
        # A thumbnail: the smallest render, a chain of short launches.
        _render("render_thumb", "render", "cornell", 0, 64, 48, 4, 8),
        # The Cornell benchmark job on the plain renderer.
        _render("render_cornell", "render", "cornell", 0, 256, 256, 16, 8),
        # A preview of a large outdoor scene on the plain renderer, odd size.
        _render("render_terrain", "render", "terrain", 768, 853, 479, 9, 16),
        # A crop of a frame (the reference's --limit) of a mesh with vertex normals, to host memory.
        _render("render_crop", "window", "mesh_smooth", 0, 640, 360, 16, 8),
        # The direct-lighting integrator, the reference's default, with glass.
        _render("render_direct", "render", "cornell", 0, 128, 128, 16, 8, direct=4),
        # The headline benchmark frame on the streaming engine.
        _render("frame_terrain", "frame", "terrain", 1024, 1920, 1080, 64, 16),
        # A batch of small jobs of uneven size in one engine run.
        {"name": "jobs_soups", "call": "jobs", "n": 50_000, "jobs": 32},
        # A scene arriving: its creation and a first batch of primary rays.
        _trace("load_soup", "soup", 200_000, 65_536, 65_536, call="load"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["trace", "trace", "trace_host", "render", "render", "window", "direct", "frame", "jobs",
                       "load"])
    if call in ("trace", "trace_host", "load"):
        scene = rng.choice(["soup", "mixed", "terrain"])
        n = _log(rng, 32, 768) if scene == "terrain" else _log(rng, 300, 600_000 if scene == "soup" else 100_000)
        rays = _log(rng, 100, {"trace": 8_000_000, "trace_host": 1_000_000, "load": 200_000}[call])
        closest = rng.choice([rays, rays, rays // 2, rng.randrange(rays + 1), 0])
        c = _trace("", scene, n, rays, closest, normals=rng.random() < 0.5, call=call)
        del c["name"]
        return c
    if call == "jobs":
        return {"call": "jobs", "n": _log(rng, 2000, 50_000), "jobs": _log(rng, 2, 32)}
    scene = rng.choice(["terrain", "soup", "cornell", "mirror", "spot_far", "mesh_smooth", "mesh_flat"]
                       + (["nested_glass"] if call in ("render", "window") else []))
    n = _log(rng, 48, 768) if scene == "terrain" else _log(rng, 1000, 300_000) if scene == "soup" else 0
    width = _log(rng, 16, 1280)
    height = max(8, int(width * rng.uniform(0.4, 1.1)))
    most = max(1, min(64, (4_000_000 if call == "direct" else 16_000_000) // (width * height)))
    spp = _log(rng, 1, most) if most > 1 else 1
    direct = rng.choice([1, 2, 4]) if call == "direct" else 0
    c = _render("", "render" if call == "direct" else call, scene, n, width, height, spp, rng.choice([4, 8, 16, 25]),
                direct)
    del c["name"]
    return c


# ---------------------------------------------------------------------------

def _scene_data(case, seed):
    kind, n = case["scene"], case["n"]
    if kind == "soup":
        if case["call"] in ("trace", "trace_host", "load"):
            # edges shrink with the count, as meshes of one size get finer
            k = (1_000_000 / max(n, 1)) ** (1 / 3)
            return scenes.random_triangles(n, seed=seed, edge_lo=0.002 * k, edge_hi=0.02 * k)
        return scenes.soup_scene(n, seed=seed)
    if kind == "mixed":
        return scenes.mixed_scene(n, n // 20, n // 20, seed=seed)
    if kind == "terrain":
        small = n < 512
        return scenes.terrain_scene(n, n_spheres=40 if small else 200, env_w=256 if small else 1024,
                                    env_h=128 if small else 512)
    return _FIXED[kind]()


def _camera(case, seed):
    rng = np.random.default_rng(seed)
    w, h, kind = case["width"], case["height"], case["scene"]
    if kind == "soup":
        return scenes.orbit_camera(w, h, rng)
    cam = {"terrain": scenes.terrain_camera, "spot_far": scenes.spot_far_camera,
           "mesh_smooth": scenes.mesh_camera, "mesh_flat": scenes.mesh_camera}.get(kind, scenes.cornell_camera)(w, h)
    cam.move(cam.pos + rng.uniform(-0.02, 0.02, 3).astype(np.float32))
    return cam


def _params(case, seed):
    if case["direct"]:
        return scenes.direct_params(case["width"], case["height"], case["spp"], seed=seed,
                                    light_samples=case["direct"])
    return sb.RenderParams(width=case["width"], height=case["height"], spp=case["spp"], min_path_len=3,
                           max_path_len=case["depth"], direct_samples=1, seed=seed)


def _rays(case, seed):
    """Origins over the scene's box with a margin, directions uniform on the sphere, no far limit."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.empty((7, n), dtype=torch.float32, device="cuda")
    lo, hi = torch.tensor([[-0.1], [-0.1], [-0.1]]), torch.tensor([[1.1], [1.1], [1.1]])
    if case["scene"] == "terrain":   # heights stay within +-0.2
        lo[2], hi[2] = -0.1, 0.5
    r[0:3] = lo.cuda() + (hi - lo).cuda() * torch.rand((3, n), generator=g, device="cuda")
    z = torch.rand(n, generator=g, device="cuda") * 2 - 1
    phi = torch.rand(n, generator=g, device="cuda") * (2 * math.pi)
    s = torch.sqrt((1 - z * z).clamp_min(0))
    r[3], r[4], r[5] = s * torch.cos(phi), s * torch.sin(phi), z
    r[6] = math.inf
    return r


def prepare(case, seed):
    call = case["call"]
    st = {"call": call}
    if call in ("trace", "trace_host", "load"):
        n = case["rays"]
        data, rays = _scene_data(case, seed), _rays(case, seed)
        st.update(n=n, closest=case["closest"], data=data)
        if call != "load":
            st["scene"] = sb.Scene(data)
        if call == "trace_host":
            st.update(rays=rays.cpu().numpy(), normals=case["normals"])
        else:
            st.update(rays=rays, prim=torch.empty(n, dtype=torch.int32, device="cuda"),
                      t=torch.empty(n, dtype=torch.float32, device="cuda"),
                      normal=torch.empty((n, 3), dtype=torch.float32, device="cuda") if case["normals"] else None)
        return st
    if call == "jobs":
        # Sizes from the batched benchmark's ranges, the same for every seed.
        size, rng, jobs = np.random.default_rng(case["jobs"]), np.random.default_rng(seed), []
        for k in range(case["jobs"]):
            n = int(round(math.exp(size.uniform(math.log(1000), math.log(case["n"])))))
            res, spp = int(size.choice(scenes.BATCH_RES)), int(size.choice(scenes.BATCH_SPP))
            jobs.append((sb.Scene(scenes.soup_scene(n, seed=seed + k)), scenes.orbit_camera(res, res, rng),
                         sb.RenderParams(res, res, spp, seed=seed + k)))
        st.update(jobs=jobs, engine=sb.Engine(sb.engine_config(max_lights=1)))
    else:
        st.update(scene=sb.Scene(_scene_data(case, seed)), camera=_camera(case, seed), params=_params(case, seed))
        if call == "window":
            w, h = case["width"], case["height"]
            out = (w // 4, h // 3, w - w // 4 - w // 5, h - h // 3 - h // 7)
            st.update(pattern=(out[0] - 2, out[1] - 2, out[2] + 4, out[3] + 4), output=out)
        if call == "frame":
            paths = (case["width"] + 4) * (case["height"] + 4) * case["spp"]
            slots = min(1 << 25, max(1 << 16, 1 << (paths // 4).bit_length()))
            st.update(jobs=[(st["scene"], st["camera"], st["params"])],
                      engine=sb.Engine(sb.engine_config(max_lights=1, slots=slots)))
    if call != "window":
        jobs = st.get("jobs") or [(None, None, st["params"])]
        st["out"] = [torch.empty((p.height, p.width, 3), dtype=torch.float32, device="cuda") for _, _, p in jobs]
    return st


def run(st):
    call = st["call"]
    if call in ("trace", "load"):
        scene = st["scene"] if call == "trace" else sb.Scene(st["data"])
        nrm = st["normal"]
        scene.trace_device(st["rays"].data_ptr(), st["n"], st["closest"], st["prim"].data_ptr(), st["t"].data_ptr(),
                           None if nrm is None else nrm.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if call == "load":
            torch.cuda.current_stream().synchronize()   # the scene goes away below
            scene.close()
        return [st["prim"], st["t"], nrm]
    if call == "trace_host":
        prim, t, nrm, counts = st["scene"].trace(st["rays"], st["closest"], want_normal=st["normals"])
        return [prim, t, nrm, [counts[k] for k in sorted(counts)]]
    if call == "render":
        st["scene"].render_device(st["camera"], st["params"], st["out"][0].data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if call == "window":
        return st["scene"].render_window(st["camera"], st["params"], st["pattern"], st["output"])[0]
    st["engine"].render(st["jobs"], device_outs=[o.data_ptr() for o in st["out"]])
    return st["out"]


def _prims(case):
    n, kind = case["n"], case["scene"]
    return {"soup": n, "mixed": n + 2 * (n // 20), "terrain": 2 * (n - 1) ** 2}.get(kind, 16)


def _scene_bytes(prims):
    """Vertices (three per triangle without sharing) and a material index, read once."""
    return 40 * prims


def _ray_flops(prims):
    """A ray's walk to its depth in the tree (three slabs, two operations and two
    comparisons each, per level) and two primitive tests of about 60 operations."""
    return 12 * max(1, math.ceil(math.log2(max(2, prims)))) + 120


def work(case):
    if case["call"] == "jobs":   # expected sizes of the drawn jobs
        paths = case["jobs"] * 28_672 * 28
        return {"bytes": case["jobs"] * (_scene_bytes(case["n"] // 4) + 12 * 28_672),
                "flops": paths * (3 * _ray_flops(case["n"] // 4) + 400)}
    prims = _prims(case)
    if "rays" in case:
        n = case["rays"]
        return {"bytes": _scene_bytes(prims) + n * (28 + 8 + (12 if case["normals"] else 0)),
                "flops": n * _ray_flops(prims) + (64 * prims if case["call"] == "load" else 0)}
    share = 0.55 * 0.52 if case["call"] == "window" else 1.0
    pixels = case["width"] * case["height"] * share
    # About 1.7 closest-hit and 0.9 shadow rays a path, and the shading of a vertex and a half.
    rays = 2.6 if not case["direct"] else 1.5 + 1.5 * case["direct"]
    return {"bytes": int(_scene_bytes(prims) + 12 * pixels),
            "flops": int(pixels * case["spp"] * (rays * _ray_flops(prims) + 400))}


def _exact_closest(data, o, d):
    """(t, unit normal) of the closest hits in 64 bits, by trying every primitive."""
    dev = o.device
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
    v = f(data.vertices)[torch.from_numpy(data.triangles.astype(np.int64)).to(dev)]
    corner = torch.cat([v[:, 0], f(data.tripars["v0"])])
    e1 = torch.cat([v[:, 1] - v[:, 0], f(data.tripars["e1"])])
    e2 = torch.cat([v[:, 2] - v[:, 0], f(data.tripars["e2"])])
    par = torch.cat([torch.zeros(len(v), dtype=torch.bool, device=dev),
                     torch.from_numpy(data.tripars["parallelogram"].astype(bool)).to(dev)])
    face = torch.linalg.cross(e2, e1)
    c, rad = f(data.spheres["center"]), f(data.spheres["radius"])
    best = torch.full((len(o),), math.inf, dtype=torch.float64, device=dev)
    nrm = torch.zeros((len(o), 3), dtype=torch.float64, device=dev)
    step = max(1, 40_000_000 // len(o))
    for k in range(0, len(corner), step):
        s = slice(k, k + step)
        # Cramer's rule on o + t d = corner + u e1 + v e2
        tv = o[:, None] - corner[None, s]
        n = face[s]
        det = d @ n.T
        q = torch.linalg.cross(tv, d[:, None].expand_as(tv))
        u = (q * e2[None, s]).sum(-1) / det
        w = -(q * e1[None, s]).sum(-1) / det
        t = -(tv * n[None]).sum(-1) / det
        ok = (u >= 0) & (w >= 0) & torch.where(par[None, s], (u <= 1) & (w <= 1), u + w <= 1) & (t > 0)
        t, i = torch.where(ok, t, math.inf).min(1)
        near = t < best
        nrm[near] = torch.nn.functional.normalize(n[i[near]], dim=1)
        best = torch.minimum(best, t)
    for k in range(0, len(c), step):
        s = slice(k, k + step)
        oo = o[:, None] - c[None, s]
        a, b = (d * d).sum(-1)[:, None], (oo * d[:, None]).sum(-1)
        disc = b * b - a * ((oo * oo).sum(-1) - rad[None, s] ** 2)
        root = disc.clamp_min(0).sqrt()
        t0, t1 = (-b - root) / a, (-b + root) / a
        t, i = torch.where(disc >= 0, torch.where(t0 > 0, t0, torch.where(t1 > 0, t1, math.inf)), math.inf).min(1)
        near = t < best
        nrm[near] = torch.nn.functional.normalize(o[near] + d[near] * t[near, None] - c[k:k + step][i[near]], dim=1)
        best = torch.minimum(best, t)
    hit = torch.isfinite(best)
    return torch.where(hit, best, 0.0), nrm


def exact(case, seed):
    """Hit distances and normals of ray queries small enough to try every
    primitive.  Images have no such value: a path's random decisions in 64
    bits are not those in 32, so its samples are other samples; ids and
    counts are whole numbers."""
    if "rays" not in case or case["closest"] * _prims(case) > 60_000_000:
        return None
    n, m = case["rays"], case["closest"]
    rays = _rays(case, seed).double()
    t = torch.zeros(n, dtype=torch.float64, device="cuda")
    nrm = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    if m:
        t[:m], nrm[:m] = _exact_closest(_scene_data(case, seed), rays[0:3, :m].T.contiguous(),
                                        rays[3:6, :m].T.contiguous())
    out = [None, t, nrm if case["normals"] else None]
    return out + [None] if case["call"] == "trace_host" else out
