"""The workloads whose speed this framework is judged by.

Each case is one thing a program using the framework does, through the calls of
`toy-path-tracing_b200/tpt.py` (the ctypes mirror of the C ABI):

* ``traverse`` — a batch of ray queries (`Scene.traverse_device`, or
  `Scene.closest_hit` for host arrays) on a sphere soup or a Cornell box:
  primary rays (coherent), bounce-like rays (incoherent), closest hit or
  occlusion with a finite range.
* ``render`` — one image (`Scene.render_device`, or `Scene.render` for a host
  image) with one of the integrators, from previews to full frames.
* ``batch`` — several uneven jobs in one call (`Context.render_batch_device`).
* ``train`` — one step of inverse rendering: the image and the gradient of the
  material parameters through `tpt.render_function()`.

Sizes are those of `bench.py` and the tests where those have one (the
1,048,576-triangle soup, the 256x256x64 Cornell box, the 2.1M-triangle grid
scene, the 64-patch Cornell box), with the sample counts of the full-frame
renders cut so that a pass stays well under two seconds; a sample's cost does
not depend on their number.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parent.parent / "toy-path-tracing_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import tpt  # noqa: E402
import tpt_scenes  # noqa: E402

SOUP_TRIS_PER_SPHERE = 256
INTEGRATORS = {"mis": tpt.INTEGRATOR_MIS, "nee": tpt.INTEGRATOR_NEE, "pt": tpt.INTEGRATOR_PT,
               "bdpt": tpt.INTEGRATOR_BDPT}


def listed():
    return [
        # bounce rays of a renderer, or a visibility service: the largest batch of the benchmark
        {"name": "traverse_incoherent_16m", "kind": "traverse", "scene": "soup", "spheres": 4096, "rays": 1 << 24,
         "coherent": False, "any_hit": False, "extras": False, "host": False},
        # occlusion of primary-like segments of finite length, a count that is no multiple of anything
        {"name": "occlusion_coherent_5m", "kind": "traverse", "scene": "soup", "spheres": 4096, "rays": 5000011,
         "coherent": True, "any_hit": True, "extras": False, "host": False},
        # picking or collision queries from host arrays on a small scene: latency of one call
        {"name": "pick_host_4097", "kind": "traverse", "scene": "cornell", "spheres": 0, "rays": 4097,
         "coherent": False, "any_hit": False, "extras": True, "host": True},
        # a large batch in host arrays, as an offline visibility tool has them: copies in and out beside the query
        {"name": "traverse_host_1m", "kind": "traverse", "scene": "soup", "spheres": 1024, "rays": 1000003,
         "coherent": True, "any_hit": False, "extras": True, "host": True},
        # a preview frame of an interactive program, image on the host: latency and launches
        {"name": "preview_97x61x1", "kind": "render", "scene": "cornell", "integrator": "mis", "width": 97,
         "height": 61, "spp": 1, "depth": 8, "n_side": 0, "tris": 0, "materials": 0, "emissive": 0, "host": True},
        # the benchmark's Cornell box (OpenPBR)
        {"name": "cornell_openpbr_256", "kind": "render", "scene": "cornell", "integrator": "mis", "width": 256,
         "height": 256, "spp": 64, "depth": 8, "n_side": 0, "tris": 0, "materials": 0, "emissive": 0, "host": False},
        # delta lights and an area light on Lambert walls: light sampling at every vertex, ragged size and spp
        {"name": "lights_lambert_nee", "kind": "render", "scene": "cornell_lights", "integrator": "nee", "width": 333,
         "height": 251, "spp": 9, "depth": 6, "n_side": 0, "tris": 0, "materials": 0, "emissive": 0, "host": False},
        # dispersive glass under MIS: long paths, the costliest BSDF
        {"name": "glass_dispersion", "kind": "render", "scene": "cornell_glass", "integrator": "mis", "width": 320,
         "height": 200, "spp": 32, "depth": 16, "n_side": 0, "tris": 0, "materials": 0, "emissive": 0, "host": False},
        # a full frame of the 2.1M-triangle scene (256 materials, 10,000 emitters)
        {"name": "large_mis_1080p", "kind": "render", "scene": "grid", "integrator": "mis", "width": 1920,
         "height": 1080, "spp": 16, "depth": 16, "n_side": 32, "tris": 2048, "materials": 256, "emissive": 10000,
         "host": False},
        # the same scene with bidirectional path tracing
        {"name": "large_bdpt_480x270", "kind": "render", "scene": "grid", "integrator": "bdpt", "width": 480,
         "height": 270, "spp": 8, "depth": 10, "n_side": 32, "tris": 2048, "materials": 256, "emissive": 10000,
         "host": False},
        # uneven jobs of one call: resolutions, spp and depths of the batched workload
        {"name": "batch_8_jobs", "kind": "batch", "jobs": 8, "spec": 4, "spp_scale": 0.25},
        # one step of inverse rendering on the 64-patch box
        {"name": "train_patches_128", "kind": "train", "width": 128, "height": 128, "spp": 16, "depth": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["traverse", "traverse", "render", "render", "render", "batch", "train"])
    if kind == "traverse":
        host = rng.random() < 0.25
        soup = rng.random() < 0.75
        any_hit = rng.random() < 0.4
        return {"kind": kind, "scene": "soup" if soup else "cornell", "spheres": _log_int(rng, 16, 4096) if soup else 0,
                "rays": _log_int(rng, 1000, 1 << 20 if host else 1 << 24), "coherent": rng.random() < 0.5,
                "any_hit": any_hit, "extras": not any_hit and rng.random() < 0.4, "host": host}
    if kind == "render":
        scene = rng.choice(["cornell", "cornell_lambert", "cornell_lights", "cornell_sky", "cornell_glass", "patches",
                            "grid", "grid"])
        integrator = rng.choice(["mis", "mis", "mis", "nee", "pt", "bdpt"])
        paths = _log_int(rng, 5000, 1 << 19 if integrator == "bdpt" else 1 << 22)
        spp = min(paths, _log_int(rng, 1, 64))
        pixels = max(1, paths // spp)
        width = max(1, int(math.sqrt(pixels * rng.uniform(0.8, 1.8))))
        grid = scene == "grid"
        return {"kind": kind, "scene": scene, "integrator": integrator, "width": width,
                "height": max(1, pixels // width), "spp": spp, "depth": rng.randint(3, 8 if integrator == "bdpt" else 16),
                "n_side": rng.randint(4, 32) if grid else 0, "tris": _log_int(rng, 64, 2048) if grid else 0,
                "materials": rng.randint(8, 256) if grid else 0, "emissive": _log_int(rng, 4, 10000) if grid else 0,
                "host": rng.random() < 0.25}
    if kind == "batch":
        case = {"kind": kind, "jobs": rng.randint(2, 8), "spec": rng.randint(5, 10 ** 6),
                "spp_scale": round(rng.uniform(0.05, 0.25), 3)}
        paths = sum(p["width"] * p["height"] * p["spp"] for p in _batch_specs(case))
        case["spp_scale"] *= min(1.0, 6e7 / paths)  # no draw costs more than the listed batch
        return case
    return {"kind": kind, "width": rng.randint(40, 200), "height": rng.randint(40, 200),
            "spp": _log_int(rng, 2, 32), "depth": rng.randint(2, 10)}


# ---------------------------------------------------------------------------
_ctx = None


def _context():
    """The one context a program keeps."""
    global _ctx
    if _ctx is None:
        _ctx = tpt.Context(torch.cuda.current_device())
        _ctx.set_gpu_build(True)
    return _ctx


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _render_scene(case, seed):
    """The scene dict of a render case."""
    s = case["scene"]
    if s == "cornell":
        return tpt_scenes.cornell_box(seed)
    if s == "cornell_lambert":
        return tpt_scenes.cornell_box(seed, tpt_scenes.LAMBERT)
    if s == "cornell_lights":
        return tpt_scenes.cornell_lights(seed)
    if s == "cornell_sky":
        return tpt_scenes.cornell_environment(seed, tpt_scenes.OPENPBR)
    if s == "cornell_glass":
        return tpt_scenes.cornell_glass(seed, dispersion=1.0)
    if s == "patches":
        return tpt_scenes.cornell_patches(seed)
    return tpt_scenes.grid_scene(seed, case["n_side"], case["tris"], case["materials"], case["emissive"])


def _upload(scene):
    return tpt.Scene(_context(), scene["meshes"], scene["instances"], materials=scene["materials"], lights=scene)


def _soup_cube(spheres):
    # the benchmark's density: 4,096 spheres in a 100^3 cube
    return 100.0 * (spheres / 4096.0) ** (1.0 / 3.0)


def _traverse_geometry(case, seed):
    """(meshes, instances, low corner, high corner) of a traverse case."""
    if case["scene"] == "soup":
        cube = _soup_cube(case["spheres"])
        mesh = tpt_scenes.sphere_soup(seed, case["spheres"], cube)
        return [mesh], [tpt_scenes.identity_instance()], (0.0, 0.0, 0.0), (cube, cube, cube)
    sc = tpt_scenes.lift_boxes(tpt_scenes.cornell_box(seed))
    return sc["meshes"], sc["instances"], (-1.4, 0.1, -1.4), (1.4, 2.9, 1.4)


def _rays(case, seed, lo, hi):
    """float32 [7, n] on the GPU: incoherent rays start uniformly in the box
    and leave in uniform directions; coherent ones are pinhole rays, four per
    pixel in pixel order.  Occlusion rays end within the box's width."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo_t = torch.tensor(lo, device="cuda", dtype=torch.float32)[:, None]
    size = torch.tensor(hi, device="cuda", dtype=torch.float32)[:, None] - lo_t
    rays = torch.empty((7, n), device="cuda", dtype=torch.float32)
    if case["coherent"]:
        side = max(1, math.ceil(math.sqrt(n / 4)))
        k = torch.arange(n, device="cuda")
        pix, sub = k // 4, k % 4
        jitter = torch.rand((2, n), generator=g, device="cuda")
        x = ((pix % side) + (sub % 2 + jitter[0]) / 2) / side * 2 - 1
        y = 1 - ((pix // side) + (sub // 2 + jitter[1]) / 2) / side * 2
        tan = math.tan(math.radians(30.0))
        rays[0:3] = lo_t + size * torch.tensor([0.5, 0.5, -0.8], device="cuda")[:, None]
        rays[3], rays[4], rays[5] = x * tan, y * tan, 1.0
    else:
        rays[0:3] = lo_t + size * torch.rand((3, n), generator=g, device="cuda")
        rays[3:6] = torch.randn((3, n), generator=g, device="cuda")
    rays[3:6] /= rays[3:6].norm(dim=0, keepdim=True)
    width = float(size.max())
    if case["any_hit"]:
        rays[6] = width * (0.05 + 1.5 * torch.rand(n, generator=g, device="cuda"))
    else:
        rays[6] = math.inf
    return rays


def _batch_specs(case):
    """Sizes of the jobs of a batch case (the same for every seed)."""
    rng = np.random.default_rng(case["spec"])
    specs = []
    for _ in range(case["jobs"]):
        tris = float(np.exp(rng.uniform(np.log(1e4), np.log(5e5))))
        n_side = int(rng.integers(4, 17))
        w, h = tpt_scenes.BATCH_RESOLUTIONS[int(rng.integers(0, len(tpt_scenes.BATCH_RESOLUTIONS)))]
        specs.append({"n_side": n_side, "tris": max(24, int(tris / (n_side * n_side))),
                      "emissive": int(np.exp(rng.uniform(np.log(4), np.log(1024)))),
                      "materials": int(rng.integers(8, 65)), "width": w, "height": h,
                      "spp": max(1, int(round(tpt_scenes.BATCH_SPP[int(rng.integers(0, 3))] * case["spp_scale"]))),
                      "depth": int(rng.integers(8, 17))})
    return specs


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "traverse":
        meshes, instances, lo, hi = _traverse_geometry(case, seed)
        st["scene"] = tpt.Scene(_context(), meshes, instances)
        rays = _rays(case, seed, lo, hi)
        st["mode"] = tpt.ANY_HIT if case["any_hit"] else tpt.CLOSEST_HIT
        st["n"], st["extras"], st["host"] = case["rays"], case["extras"], case["host"]
        if case["host"]:
            st["rays"] = rays.cpu().numpy()
        else:
            st["rays"] = rays
            st["prim"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
            st["t"] = torch.empty(case["rays"], dtype=torch.float32, device="cuda")
            if case["extras"]:
                st["inst"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
                st["bary"] = torch.empty((3, case["rays"]), dtype=torch.float32, device="cuda")
    elif kind == "render":
        sc = _render_scene(case, seed)
        st["scene"], st["camera"], st["host"] = _upload(sc), sc["camera"], case["host"]
        st["args"] = (case["width"], case["height"], case["spp"], case["depth"], INTEGRATORS[case["integrator"]],
                      tpt.EXEC_WAVEFRONT, seed & 0xFFFF)
        if not case["host"]:
            st["job"] = st["scene"].job(st["camera"], *st["args"])
            st["image"] = torch.empty((case["height"], case["width"], 3), dtype=torch.float32, device="cuda")
    elif kind == "batch":
        st["scenes"], st["jobs"], st["images"] = [], [], []
        for k, p in enumerate(_batch_specs(case)):
            sc = tpt_scenes.grid_scene(1000 * (seed % 100000) + k, p["n_side"], p["tris"], p["materials"], p["emissive"])
            up = _upload(sc)
            st["scenes"].append(up)
            st["jobs"].append(up.job(sc["camera"], p["width"], p["height"], p["spp"], p["depth"], seed=seed & 0xFFFF))
            st["images"].append(torch.empty((p["height"], p["width"], 3), dtype=torch.float32, device="cuda"))
    else:
        sc = tpt_scenes.cornell_patches(seed)
        st["scene"] = _upload(sc)
        st["job"] = st["scene"].job(sc["camera"], case["width"], case["height"], case["spp"], case["depth"],
                                    seed=seed & 0xFFFF)
        start = tpt_scenes.patch_params(seed, start=True)
        st["params"] = torch.from_numpy(start).requires_grad_(True)
        st["ids"] = np.arange(tpt_scenes.N_PATCH_MATERIALS, dtype=np.uint32)
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["d_image"] = torch.randn((case["height"], case["width"], 3), generator=g, device="cuda")
        st["render"] = tpt.render_function().apply
    return st


def run(state):
    kind = state["kind"]
    if kind == "traverse":
        if state["host"]:
            return state["scene"].closest_hit(state["rays"], state["mode"], want_instance=state["extras"],
                                              want_bary=state["extras"])
        out = {"prim": state["prim"], "t": state["t"]}
        if state["extras"]:
            out["inst"], out["bary"] = state["inst"], state["bary"]
        state["scene"].traverse_device(state["rays"].data_ptr(), state["n"], state["mode"], state["prim"].data_ptr(),
                                       state["t"].data_ptr(), state["inst"].data_ptr() if state["extras"] else None,
                                       state["bary"].data_ptr() if state["extras"] else None, _stream())
        return out
    if kind == "render":
        if state["host"]:
            return {"image": state["scene"].render(state["camera"], *state["args"])}
        state["scene"].render_device(state["job"], state["image"].data_ptr(), _stream())
        return {"image": state["image"]}
    if kind == "batch":
        _context().render_batch_device(state["jobs"], [im.data_ptr() for im in state["images"]], _stream())
        return {"images": state["images"]}
    image = state["render"](state["params"], state["scene"], state["job"], state["ids"], tpt_scenes.patch_material)
    (grad,) = torch.autograd.grad(image, state["params"], state["d_image"])
    return {"image": image, "grad": grad}


# ---------------------------------------------------------------------------
def _scene_tris(case):
    """Triangles a ray of the case may meet, distinct triangle records, instances."""
    s = case["scene"]
    if s == "soup":
        n = case["spheres"] * SOUP_TRIS_PER_SPHERE
        return n, n, 1
    if s == "patches":
        return 2018, 2018, 65
    if s == "grid":
        emit = 2 * max(1, case["emissive"] // 2)
        objects = case["n_side"] ** 2
        return objects * case["tris"] + emit, 3 * case["tris"] + 4, objects + emit // 2 + 1
    return 36, 24, 8


def _ray_flops(tris):
    """Least arithmetic of one closest-hit query: one 4-wide slab test (4 x 22)
    per level of a 4-wide tree and two triangle tests of about 60."""
    return 88.0 * max(1.0, math.log(max(tris, 4), 4)) + 120.0


# arithmetic of one shading vertex (BSDF value, density and sample, light
# sample, random numbers), a round figure
VERTEX_FLOPS = 400.0


def _render_work(case):
    tris, records, instances = _scene_tris(case)
    samples = float(case["width"]) * case["height"] * case["spp"]
    rays = min(case["depth"] + 1, 4) * (2 if case["integrator"] in ("mis", "nee") else 1)
    if case["integrator"] == "bdpt":
        rays = 8 + 16  # two subpaths of about four vertices and their connections
    return {"bytes": 12.0 * case["width"] * case["height"] + 60.0 * records + 64.0 * instances,
            "flops": samples * rays * (_ray_flops(tris) + VERTEX_FLOPS)}


def work(case):
    kind = case["kind"]
    if kind == "traverse":
        tris, records, instances = _scene_tris(case)
        per_ray = (28 if case["any_hit"] else 24) + 8 + (16 if case["extras"] else 0)
        return {"bytes": float(case["rays"]) * per_ray + 60.0 * records + 64.0 * instances,
                "flops": case["rays"] * _ray_flops(tris)}
    if kind == "render":
        return _render_work(case)
    if kind == "batch":
        parts = [_render_work(dict(p, scene="grid", integrator="mis")) for p in _batch_specs(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    one = _render_work(dict(case, scene="patches", integrator="mis"))
    # forward, replay, and two perturbed BSDF values per parameter group
    return {"bytes": 2 * one["bytes"], "flops": 4 * one["flops"]}


def exact(case, seed):
    """Hit distances and barycentrics of the nearest triangle by brute force in
    64 bits, for the query batches small enough for it.  Which hit an occlusion
    query reports is the traversal's choice, and a rendered image depends on
    every 32-bit decision of its paths: neither has a 64-bit value."""
    if case["kind"] != "traverse" or case["any_hit"]:
        return None
    tris = _scene_tris(case)[0]
    if case["rays"] * tris > 3_000_000_000:
        return None
    meshes, instances, lo, hi = _traverse_geometry(case, seed)
    rays = _rays(case, seed, lo, hi).double()
    corners = []
    for inst in instances:
        m = torch.from_numpy(np.asarray(inst["local_to_world"], np.float64).reshape(4, 4).T.copy()).cuda()
        mesh = meshes[inst["mesh"]]
        p = torch.from_numpy(mesh["positions"].astype(np.float64)).cuda() @ m[:3, :3].T + m[:3, 3]
        corners.append(p[torch.from_numpy(mesh["indices"].astype(np.int64)).cuda()].view(-1, 3, 3))
    tri = torch.cat(corners)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    # with n = e1 x e2 and the scalar triple products of Moeller and Trumbore
    n = torch.linalg.cross(e1, e2)
    ts, bs = [], []
    step = max(1, 20_000_000 // max(1, tri.shape[0]))
    for k in range(0, case["rays"], step):
        o, d = rays[0:3, k:k + step].T, rays[3:6, k:k + step].T
        det = -(d @ n.T)
        # (o - v0) . n, and u, v through (o - v0) x d = o x d - v0 x d
        num = o @ n.T - (v0 * n).sum(1)
        od = torch.linalg.cross(o, d)
        u = od @ e2.T - d @ torch.linalg.cross(e2, v0).T
        v = -(od @ e1.T) + d @ torch.linalg.cross(e1, v0).T
        t, u, v = num / det, u / det, v / det
        hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-9)
        t = torch.where(hit, t, math.inf)
        best = t.argmin(1, keepdim=True)
        tb = t.gather(1, best)[:, 0]
        ub, vb = u.gather(1, best)[:, 0], v.gather(1, best)[:, 0]
        b = torch.stack([1 - ub - vb, ub, vb])
        ts.append(tb)
        bs.append(torch.where(torch.isfinite(tb)[None], b, 0.0))
    out = {"prim": None, "t": torch.cat(ts)}
    if case["extras"]:
        out["inst"], out["bary"] = None, torch.cat(bs, 1)
    return out
