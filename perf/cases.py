"""Performance cases: what a program that uses this renderer has it do.

Every case goes through the package's public entry points (HostScene, Renderer, guide_train) on
the repository's own procedural scenes (xenon_b200/scenes.py): the Cornell box of config 1, the
displaced icosphere of config 2, the instanced grid of config 3 and the guided room of config 4,
at those configurations' sizes and below. Kinds of case:

  query    ray queries, from host arrays (picking, placement) or device arrays (baking, physics)
  render   samples of one view into the framebuffer, and the image back on the host
  views    several views of different sizes in one call (config 5)
  animate  a mesh's vertices move: BLAS refit, one sample of every pixel, the image back
  load     BVH build on the device and upload, with a first picking query
  fit      the guiding network trained further on a set of records

`listed()` are fixed cases, `draw(rng)` gives more from the same ranges.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import xenon_b200 as xb
from xenon_b200 import abi, autotune, scenes

PATHS_MAX = 1920 * 1080 * 8   # paths of the largest listed render (icosphere)
GRID_PATHS_MAX = 1920 * 1080 * 2
ROOM_PATHS_MAX = 1280 * 720 * 4


def listed() -> list:
    return [
        # an editor's pick or a placement test: a handful of rays from host memory, answer wanted now
        {"name": "query_pick_host", "kind": "query", "scene": "cornell", "size": 0, "rays": 1000,
         "spread": "uniform", "mode": "closest", "host": True},
        # light baking or simulation: a large incoherent batch that lives on the device
        {"name": "query_uniform_device", "kind": "query", "scene": "icosphere", "size": 8, "rays": 1 << 22,
         "spread": "uniform", "mode": "closest", "host": False},
        # ambient occlusion over an instanced scene: any-hit rays off its surfaces, a ragged count
        {"name": "query_occlusion_device", "kind": "query", "scene": "grid", "size": 16, "rays": 1000003,
         "spread": "hemisphere", "mode": "any", "host": False},
        # interactive preview: one sample per pixel per displayed frame, default settings (config 1)
        {"name": "frame_cornell_256", "kind": "render", "scene": "cornell", "size": 0, "width": 256,
         "height": 256, "spp": 1, "tuning": "", "guided": False, "out": "image"},
        # an offline still of the same box at its configured sample count, written as a PNG's pixels
        {"name": "still_cornell_256_64spp", "kind": "render", "scene": "cornell", "size": 0, "width": 256,
         "height": 256, "spp": 64, "tuning": "", "guided": False, "out": "stage"},
        # the headline render: config 2 at full size with its stored tuning, image by resolve_async
        {"name": "still_icosphere_1080p_8spp", "kind": "render", "scene": "icosphere", "size": 8,
         "width": 1920, "height": 1080, "spp": 8, "tuning": "config2", "guided": False, "out": "pinned"},
        # config 3 (instances, all material kinds) at full size with its stored tuning
        {"name": "still_grid_1080p_2spp", "kind": "render", "scene": "grid", "size": 16, "width": 1920,
         "height": 1080, "spp": 2, "tuning": "config3", "guided": False, "out": "image"},
        # config 4 guided by a network that is held fixed, stored tuning
        {"name": "guided_room_720p_4spp", "kind": "render", "scene": "room", "size": 158, "width": 1280,
         "height": 720, "spp": 4, "tuning": "config4g", "guided": True, "out": "image"},
        # config 5: a few small views of odd sizes and depths packed together
        {"name": "views_grid_6", "kind": "views", "scene": "grid", "size": 8, "views": 6, "side_min": 160,
         "side_max": 420, "spp": 8},
        # an animated mesh: refit, one sample, image
        {"name": "animate_icosphere_540p", "kind": "animate", "size": 7, "width": 960, "height": 540},
        # opening a scene: BVH build on the device, upload, first pick
        {"name": "load_icosphere_1300k", "kind": "load", "size": 8},
        # continued training of the guiding network on records of a scene
        {"name": "fit_guide_128_steps", "kind": "fit", "records": 200000, "steps": 128, "batch": 16384},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["query", "query", "query", "render", "render", "render", "render", "views", "animate",
                       "load", "fit"])
    scene = rng.choice(["cornell", "icosphere", "grid", "room"])
    size = {"cornell": 0, "icosphere": rng.randint(3, 8), "grid": rng.randint(2, 16),
            "room": rng.randint(20, 158)}[scene]
    if kind == "query":
        rays = _log_int(rng, 1000, 1 << 22) if scene in ("cornell", "icosphere") else _log_int(rng, 1000, 1000003)
        host = rays <= 200000 and rng.random() < 0.4
        return {"kind": kind, "scene": scene, "size": size, "rays": rays,
                "spread": rng.choice(["uniform", "hemisphere"]), "mode": rng.choice(["closest", "any"]), "host": host}
    if kind == "render":
        width = _log_int(rng, 48, 1920)
        height = max(27, min(1080, int(width * rng.uniform(0.5, 1.0))))
        cap = {"cornell": PATHS_MAX // 4, "icosphere": PATHS_MAX, "grid": GRID_PATHS_MAX, "room": ROOM_PATHS_MAX}[scene]
        spp = _log_int(rng, 1, max(1, min(64, cap // (width * height))))
        guided = scene in ("room", "grid") and rng.random() < 0.4
        tuning = rng.choice(["", {"cornell": "", "icosphere": "config2", "grid": "config3",
                                  "room": "config4g" if guided else "config4"}[scene]])
        return {"kind": kind, "scene": scene, "size": size, "width": width, "height": height, "spp": spp,
                "tuning": tuning, "guided": guided, "out": rng.choice(["image", "stage", "pinned"])}
    if kind == "views":
        lo = _log_int(rng, 64, 200)
        return {"kind": kind, "scene": "grid", "size": rng.randint(2, 8), "views": rng.randint(1, 6),
                "side_min": lo, "side_max": _log_int(rng, lo, 420), "spp": _log_int(rng, 1, 8)}
    if kind == "animate":
        width = _log_int(rng, 64, 960)
        return {"kind": kind, "size": rng.randint(3, 7), "width": width,
                "height": max(36, int(width * rng.uniform(0.4, 0.5625)))}
    if kind == "load":
        return {"kind": kind, "size": rng.randint(2, 8)}
    return {"kind": kind, "records": _log_int(rng, 3000, 200000), "steps": _log_int(rng, 8, 128),
            "batch": 128 * _log_int(rng, 1, 128)}


# ── scenes (their geometry is made once per process, as a program loads its assets once) ──────
@functools.lru_cache(maxsize=8)
def _desc(scene: str, size: int):
    if scene == "cornell":
        return scenes.cornell()
    if scene == "icosphere":
        return scenes.icosphere_scene(level=size)
    if scene == "grid":
        return scenes.instanced_grid(grid=size)
    return scenes.guiding_room(freq=size)


@functools.lru_cache(maxsize=4)
def _host_scene(scene: str, size: int):
    return xb.HostScene.from_desc(_desc(scene, size))


def _camera(desc, seed: int, width: int, height: int):
    rng = np.random.default_rng(seed)
    eye = np.asarray(desc.eye, np.float64) + rng.uniform(-0.1, 0.1, 3)
    return xb.camera(eye, desc.target, desc.fov, width / height)


def _moved(desc, seed: int):
    """The largest mesh's index and its vertices under a smooth seeded displacement of a few percent."""
    m = int(np.argmax([len(x.positions) for x in desc.meshes]))
    pos = np.asarray(desc.meshes[m].positions, np.float64)
    rng = np.random.default_rng(seed)
    f, ph = rng.uniform(0.5, 2.0, (3, 3)), rng.uniform(0, 2 * np.pi, 3)
    amp = 0.02 * float(np.abs(pos[:-4]).max()) if len(pos) > 4 else 0.02
    return m, (pos + amp * np.sin(pos @ f + ph)).astype(np.float32)


def _uniform_rays(view, n: int, seed: int) -> torch.Tensor:
    """Origins uniform in the scene's bounds, directions uniform on the sphere: float32 [n, 8]."""
    lo, hi = (torch.tensor(b, dtype=torch.float32, device="cuda") for b in _root_box(view))
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = torch.randn(n, 3, generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty(n, 8, device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda")
    rays[:, 3] = 1e-4
    rays[:, 4:7] = d
    rays[:, 7] = float("inf")
    return rays


def _root_box(view):
    root = np.frombuffer((ctypes.c_char * 32).from_address(view.tlas_nodes), abi.NODE_DTYPE)[0]
    return root["mn"].tolist(), root["mx"].tolist()


def _hemisphere_rays(r, desc, n: int, seed: int) -> torch.Tensor:
    """Cosine-distributed rays off the surfaces that a view of the scene sees (what ambient
    occlusion traces): camera rays are traced, then each hit sends rays about its normal."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = _camera(desc, seed, 16, 9).to_array().astype(np.float32)
    eye, ll, hor, ver = (torch.tensor(c[k:k + 3], device="cuda") for k in (0, 3, 6, 9))
    m = 65536
    uv = torch.rand(m, 2, generator=g, device="cuda")
    d = ll + uv[:, :1] * hor + uv[:, 1:] * ver - eye
    cam = torch.empty(m, 8, device="cuda")
    cam[:, 0:3], cam[:, 3] = eye, 1e-4
    cam[:, 4:7], cam[:, 7] = d / d.norm(dim=1, keepdim=True), float("inf")
    hits = torch.empty(m, 16, device="cuda")
    torch.cuda.synchronize()
    r.trace_rays_device(cam.data_ptr(), m, hits.data_ptr(), abi.XB_TRACE_CLOSEST)
    torch.cuda.synchronize()
    hits = hits[torch.isfinite(hits[:, 0])]
    pick = torch.randint(len(hits), (n,), generator=g, device="cuda")
    pos, nrm = hits[pick, 7:10], hits[pick, 13:16]
    nrm = torch.where((nrm * cam[0, 4:7]).sum(1, keepdim=True) > 0, -nrm, nrm)
    v = torch.randn(n, 3, generator=g, device="cuda")
    v = nrm + v / v.norm(dim=1, keepdim=True) * 0.999
    rays = torch.empty(n, 8, device="cuda")
    rays[:, 0:3], rays[:, 3] = pos + 1e-3 * nrm, 1e-4
    rays[:, 4:7], rays[:, 7] = v / v.norm(dim=1, keepdim=True), float("inf")
    return rays


def _views(case: dict, seed: int) -> list:
    """Cameras as config 5 draws them: square views from the upper hemisphere, depths 6 to 16."""
    desc = _desc(case["scene"], case["size"])
    lo, hi = (np.asarray(b, np.float64) for b in scenes.scene_bounds(desc))
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["views"])   # the sizes are the case's, the cameras the seed's
    out = []
    for _ in range(case["views"]):
        d = rng.normal(size=3)
        d[1] = abs(d[1]) + 0.3
        eye = (lo + hi) / 2 + d / np.linalg.norm(d) * np.linalg.norm(hi - lo) / 2 * rng.uniform(0.6, 1.2)
        side = int(sizes.integers(case["side_min"], case["side_max"] + 1))
        out.append((xb.camera(eye, (lo + hi) / 2, 45.0, 1.0), side, side, case["spp"], int(sizes.integers(6, 17))))
    return out


def _guide_params(seed: int) -> np.ndarray:
    p = xb.guide_init_params(seed + 1)
    p[3 * 4160:] *= 10.0   # distinct lobes, as after training
    return p


def _records(n: int, seed: int) -> np.ndarray:
    """Training records: features, direction, weight and BSDF density (24 floats each)."""
    rng = np.random.default_rng(seed)
    unit = rng.standard_normal((3, n, 3)).astype(np.float32)
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    rec = np.zeros((n, 24), np.float32)
    rec[:, 0:3] = rng.random((n, 3), dtype=np.float32)
    rec[:, 3:6], rec[:, 6:9] = unit[0], unit[1]
    # light arrives mostly from one side of the unit box, as it does in a room
    toward = np.float32([0.8, 1.0, 0.3]) - rec[:, 0:3] + 0.4 * unit[2]
    rec[:, 9:12] = toward / np.linalg.norm(toward, axis=1, keepdims=True)
    rec[:, 12] = rng.exponential(1.0, n)
    rec[:, 20] = rng.random(n, dtype=np.float32) * 0.5
    return rec


# ── prepare / run ────────────────────────────────────────────────────────────────────
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "query":
        desc, hs = _desc(case["scene"], case["size"]), _host_scene(case["scene"], case["size"])
        r = xb.Renderer(64, 64)
        r.upload_scene(hs)
        rays = (_uniform_rays(hs.view(), case["rays"], seed) if case["spread"] == "uniform"
                else _hemisphere_rays(r, desc, case["rays"], seed))
        st["mode"] = abi.XB_TRACE_CLOSEST if case["mode"] == "closest" else abi.XB_TRACE_ANY
        if case["host"]:
            st["rays"] = rays.cpu().numpy().view(abi.RAY_DTYPE).reshape(-1)
        else:
            st["rays"], st["hits"] = rays, torch.empty(case["rays"], 16, device="cuda")
            st["stream"] = torch.cuda.Stream()
    elif kind == "render":
        desc = _desc(case["scene"], case["size"])
        r = xb.Renderer(case["width"], case["height"], desc.max_bounces, desc.min_bounces)
        tuning = autotune.load_tuning(case["tuning"]) if case["tuning"] else None
        if tuning:
            r.set_tuning(**tuning)
        r.upload_scene(_host_scene(case["scene"], case["size"]))
        if case["guided"]:
            r.set_guiding(True, train_spp=-1)
            r.set_guide_params(_guide_params(seed))
        st["camera"] = _camera(desc, seed, case["width"], case["height"])
        if case["out"] == "pinned":
            st["pinned"] = torch.empty(case["height"], case["width"], 3, pin_memory=True)
    elif kind == "views":
        desc = _desc(case["scene"], case["size"])
        r = xb.Renderer(64, 64, desc.max_bounces, desc.min_bounces)
        r.upload_scene(_host_scene(case["scene"], case["size"]))
        st["views"] = _views(case, seed)
    elif kind == "animate":
        desc = _desc("icosphere", case["size"])
        r = xb.Renderer(case["width"], case["height"], desc.max_bounces, desc.min_bounces)
        r.upload_scene(_host_scene("icosphere", case["size"]))
        st["mesh"], st["positions"] = _moved(desc, seed)
        st["camera"] = _camera(desc, 0, case["width"], case["height"])
    elif kind == "load":
        base = _desc("icosphere", case["size"])
        mesh, pos = _moved(base, seed)
        desc = scenes.SceneDesc(**{**base.__dict__, "meshes": list(base.meshes)})
        desc.meshes[mesh] = scenes.MeshDesc(**{**base.meshes[mesh].__dict__, "positions": pos})
        st["scene"] = xb.HostScene.from_desc(desc, build=False)
        tris = base.num_triangles
        st["nodes"], st["order"] = np.zeros((2 * tris, 8), np.int32), np.zeros(tris, np.int32)
        r = xb.Renderer(64, 64)
        rng = np.random.default_rng(seed)
        d = rng.normal(size=(256, 3))
        st["rays"] = abi.make_rays(np.tile(np.float32(desc.eye), (256, 1)),
                                   (np.float32([0, -0.1, -1]) + 0.1 * d).astype(np.float32))
    else:
        r = None
        st["params"], st["records"], st["seed"] = _guide_params(seed), _records(case["records"], seed), seed + 1
    st["renderer"] = r
    torch.cuda.synchronize()
    return st


def _hit_fields(hits) -> dict:
    """The fields of hit records: float32 [n, 16] on the device, or an array of abi.HIT_DTYPE."""
    if isinstance(hits, torch.Tensor):
        f, ids = hits, hits.view(torch.int32)
    else:
        f = hits.view(np.float32).reshape(-1, 16)
        ids = f.view(np.int32)
    return {"t": f[:, 0], "uv": f[:, 1:3], "ids": ids[:, 3:7], "pos": f[:, 7:10], "normal": f[:, 10:13],
            "geo_normal": f[:, 13:16]}


def run(st: dict):
    case, r = st["case"], st["renderer"]
    kind = case["kind"]
    if kind == "query":
        if case["host"]:
            return _hit_fields(r.trace_rays(st["rays"], st["mode"]))
        r.trace_rays_device(st["rays"].data_ptr(), case["rays"], st["hits"].data_ptr(), st["mode"],
                            st["stream"].cuda_stream)
        return _hit_fields(st["hits"])
    if kind == "render":
        r.reset()
        r.render_frame(st["camera"], case["spp"])
        if case["out"] == "stage":
            pixels, stats = r.output_stage()
            return {"pixels": pixels, "stats": stats, "image": r.resolve()}
        if case["out"] == "pinned":
            r.resolve_async(st["pinned"].numpy())
            r.sync()
            return st["pinned"]
        return r.resolve()
    if kind == "views":
        return r.render_views(st["views"])
    if kind == "animate":
        r.refit_mesh(st["mesh"], st["positions"])
        r.reset()
        r.render_frame(st["camera"], 1)
        return r.resolve()
    if kind == "load":
        hs = st["scene"]
        hs.build(build_mode=abi.XB_BUILD_DEVICE)
        r.upload_scene(hs)
        hits = r.trace_rays(st["rays"])
        # the tree as a program keeps it to be written to a cache file
        mv = hs.view().meshes[0]
        ctypes.memmove(st["nodes"].ctypes.data, mv.blas_nodes, 32 * mv.num_blas_nodes)
        st["nodes"][mv.num_blas_nodes:] = 0
        ctypes.memmove(st["order"].ctypes.data, mv.blas_prims, 4 * mv.num_triangles)
        return {"nodes": st["nodes"], "order": st["order"], "hits": _hit_fields(hits)}
    params, losses = xb.guide_train(st["params"], st["records"], case["steps"], case["batch"], lr=5e-4,
                                    seed=st["seed"])
    return {"params": params, "losses": losses}


# ── work ─────────────────────────────────────────────────────────────────────────────
def _triangles(scene: str, size: int) -> int:
    return {"cornell": 36, "icosphere": 20 * 4 ** size + 2, "grid": 3 * 20 * (2 * 4 ** 6 + 2 * 4 ** 7) + 10,
            "room": 20 * size * size + 18}[scene]


def work(case: dict) -> dict:
    """Bytes: rays or pixels and the scene's triangles (36 B) and nodes (32 B each, one per
    triangle) once. Flops: 30 per node of one root-to-leaf descent (two slab tests) and 40 per
    leaf triangle for every ray; 200 per shaded path vertex; the network's multiply-adds."""
    kind = case["kind"]
    if kind == "fit":
        rows = case["steps"] * case["batch"]
        return {"bytes": case["records"] * 96 + 2 * 4 * 15600, "flops": rows * (30720 + 22528 + 30720)}
    scene, size = case.get("scene", "icosphere"), case["size"]
    tris = _triangles(scene, size)
    per_ray = 30 * math.log2(tris) + 40
    scene_bytes = 68 * tris
    if kind == "query":
        return {"bytes": case["rays"] * (32 + 64) + scene_bytes, "flops": case["rays"] * per_ray}
    if kind == "load":
        return {"bytes": tris * (36 + 32 + 4) * 2, "flops": tris * math.log2(tris) * 30}
    # rays and shaded vertices per path, as counted on these scenes
    rays, verts = {"cornell": (9.0, 5.0), "icosphere": (2.4, 1.4), "grid": (3.0, 2.0), "room": (16.0, 8.0)}[scene]
    if kind == "views":
        side = (case["side_min"] + case["side_max"]) / 2
        pixels, spp = case["views"] * side * side, case["spp"]
    else:
        pixels, spp = case["width"] * case["height"], case.get("spp", 1)
    flops = pixels * spp * (rays * per_ray + verts * (200 + (30720 if case.get("guided") else 0)))
    return {"bytes": pixels * 12 + scene_bytes, "flops": flops}


# ── exact values ─────────────────────────────────────────────────────────────────────
def exact(case: dict, seed: int):
    """Closest hits of a query by brute force over the triangles in FP64, where that is quick (the
    Cornell box and the smaller icospheres, whose instances are identities). Two quads of the
    Cornell box coincide, so which of them a hit is on, and with it u, v and the normals, has no
    exact value there; shading normals are the mesh's own. The other outputs have none either: a
    path's image depends on every branch its 32-bit arithmetic takes, training on the sums' order,
    and any-hit answers and trees hold no computed numbers."""
    if case["kind"] != "query" or case["mode"] != "closest" or case["scene"] not in ("cornell", "icosphere"):
        return None
    tris = _triangles(case["scene"], case["size"])
    if case["rays"] * tris > 2e10:
        return None
    rays = prepare(case, seed)["rays"]
    rays = (torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()) if case["host"] else rays).double().cuda()
    p = np.concatenate([m.positions[m.indices] for m in _desc(case["scene"], case["size"]).meshes])
    p0, p1, p2 = torch.from_numpy(p.astype(np.float64)).cuda().unbind(1)
    e1, e2 = p1 - p0, p2 - p0
    out = {"t": [], "uv": [], "pos": [], "geo_normal": []}
    for ray in rays.split(max(1, (1 << 25) // tris)):
        o, d = ray[:, None, 0:3], ray[:, None, 4:7]
        h = torch.linalg.cross(d, e2[None])
        inv = 1.0 / (e1 * h).sum(-1)
        s = o - p0
        u = (s * h).sum(-1) * inv
        q = torch.linalg.cross(s, e1[None])
        v = (d * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        ok = torch.isfinite(inv) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= ray[:, 3:4])
        t, tri = torch.where(ok, t, torch.inf).min(1)
        miss = ~torch.isfinite(t)
        g = torch.linalg.cross(e1[tri], e2[tri])
        uv = torch.stack([u.gather(1, tri[:, None])[:, 0], v.gather(1, tri[:, None])[:, 0]], 1)
        pos = ray[:, 0:3] + torch.where(miss, 0.0, t)[:, None] * ray[:, 4:7]
        for k, x in (("uv", uv), ("pos", pos), ("geo_normal", g / g.norm(dim=1, keepdim=True))):
            out[k].append(torch.where(miss[:, None], 0.0, x))
        out["t"].append(t)
    out = {k: torch.cat(x) for k, x in out.items()}
    if case["scene"] == "cornell":
        out["uv"] = out["geo_normal"] = None
    return {**out, "ids": None, "normal": None}
