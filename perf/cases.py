"""The work that users of the ray-query library have it do, as timed cases.

Each case is one call (or the short sequence of calls) that a program makes
per query, frame, optimisation step or model load, through the public Python
binding of the C interface: single and batched host queries (ISceneObject),
device-resident frames of meshes and SDF models, the host-buffer frame, many
cameras at once, a primary + diffuse-bounce wavefront, the differentiable
render's step, the fused renderer, an animated scene and a mesh load.

Scenes come from the package's seeded generators and stay loaded between
calls, as a renderer keeps them; the seed moves the camera a little (the next
frame of a camera path), or draws the rays, poses, colours, values or mesh that
the call takes.
"""
import functools
import math

import numpy as np
import torch

from graphic_lab_task_b200 import (BUILD_LOW, LIGHT_AMBIENT, LIGHT_DIRECT, LIGHT_DTYPE, LIGHT_POINT, MATERIAL_COLORED,
                                   MATERIAL_DTYPE, SceneRT, default_preset, parity_preset, workloads as wl)
from graphic_lab_task_b200._abi import SBS_LAYOUT_DX
from graphic_lab_task_b200.lrt import CameraBatch

TNEAR, TFAR = 1e-4, 100.0
BACKGROUND = (0.1, 0.2, 0.3, 1.0)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a picking or collision query: one ray from the host, one answer back
        {"name": "query_one", "kind": "query", "scene": "mesh", "size": 50000},
        # visibility queries of a host program: a few thousand unsorted rays in ordinary memory
        {"name": "host_rays_4k", "kind": "host_batch", "scene": "mesh", "size": 200000, "rays": 4099},
        # a small preview frame of a mesh, rays resident, row order
        {"name": "mesh_frame_256", "kind": "frame", "scene": "mesh", "size": 200000, "width": 256, "height": 256,
         "order": "row"},
        # a window of odd size on a sparse voxel set under the renderer's default preset (ANALYTIC node solver)
        {"name": "svs_frame_odd", "kind": "frame", "scene": "svs", "size": 7, "width": 1001, "height": 777,
         "order": "image"},
        # the full-HD frame of a 512^3 sparse brick set: G-buffer of an interactive viewer
        {"name": "sbs_frame_1080p", "kind": "frame", "scene": "sbs", "size": 512, "width": 1920, "height": 1080,
         "order": "image"},
        # the same frame for a host program: pinned rays in, pinned hits out
        {"name": "sbs_host_1080p", "kind": "host_frame", "scene": "sbs", "size": 512, "width": 1920, "height": 1080},
        # offline rendering of one model from many cameras of mixed resolutions
        {"name": "cameras_64", "kind": "cameras", "scene": "sbs", "size": 512, "cameras": 64, "res_min": 128,
         "res_max": 2048},
        # path tracing's first two wavefronts on a two-level scene: primary rays and one diffuse bounce
        {"name": "wavefront_4096", "kind": "wavefront", "scene": "instanced", "size": 1024, "depth": 8, "side": 4096},
        # an optimisation step over an SDF's values: new values, forward images, gradients
        {"name": "lambert_step_256", "kind": "lambert_step", "size": 256, "views": 16, "res": 512},
        # the renderer with coloured, partly transparent materials on a scene of all four geometry kinds
        {"name": "render_mixed_720p", "kind": "render", "scene": "mixed", "size": 24, "width": 1280, "height": 720,
         "mode": 17, "spp": 1, "alpha": 0.5},
        # an animated scene: every instance moves, the scene is committed, a frame is rendered
        {"name": "animate_256", "kind": "animate", "scene": "moving", "size": 256, "width": 1280, "height": 720},
        # a mesh loaded with the fast build, up to its first frame
        {"name": "load_mesh_500k", "kind": "load", "size": 500000, "width": 512, "height": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "host_batch", "frame", "frame", "frame", "host_frame", "cameras", "wavefront",
                       "lambert_step", "render", "animate", "load"])
    if kind == "query":
        scene = rng.choice(["mesh", "sbs", "svs"])
        return {"kind": kind, "scene": scene, "size": _size(rng, scene)}
    if kind == "host_batch":
        scene = rng.choice(["mesh", "sbs", "svs"])
        return {"kind": kind, "scene": scene, "size": _size(rng, scene), "rays": _log(rng, 2, 200000)}
    if kind in ("frame", "host_frame"):
        scene = rng.choice(["mesh", "sbs", "svs"] if kind == "frame" else ["mesh", "sbs"])
        c = {"kind": kind, "scene": scene, "size": _size(rng, scene), "width": _log(rng, 48, 2560),
             "height": _log(rng, 40, 1440)}
        if kind == "frame":
            c["order"] = rng.choice(["image", "image", "row"])
        return c
    if kind == "cameras":
        return {"kind": kind, "scene": "sbs", "size": _size(rng, "sbs"), "cameras": _log(rng, 2, 40),
                "res_min": _log(rng, 32, 200), "res_max": _log(rng, 256, 1800)}
    if kind == "wavefront":
        return {"kind": kind, "scene": "instanced", "size": _log(rng, 32, 1024), "depth": rng.choice([6, 7]),
                "side": _log(rng, 128, 3500)}
    if kind == "lambert_step":
        return {"kind": kind, "size": 8 * rng.randint(8, 32), "views": _log(rng, 1, 16), "res": _log(rng, 65, 512)}
    if kind == "render":
        return {"kind": kind, "scene": "mixed", "size": rng.randint(4, 40), "width": _log(rng, 64, 1920),
                "height": _log(rng, 48, 1080), "mode": rng.choice([1, 17, 17, 16]), "spp": rng.choice([1, 1, 4]),
                "alpha": rng.choice([0.25, 0.5, 1.0])}
    if kind == "animate":
        return {"kind": kind, "scene": "moving", "size": _log(rng, 2, 512), "width": _log(rng, 64, 1920),
                "height": _log(rng, 48, 1080)}
    return {"kind": "load", "size": _log(rng, 500, 500000), "width": _log(rng, 64, 1024), "height": _log(rng, 64, 1024)}


def _size(rng, scene):
    return {"mesh": lambda: _log(rng, 2000, 500000), "sbs": lambda: 8 * rng.randint(8, 64),
            "svs": lambda: rng.choice([5, 6, 7])}[scene]()


# ---------------------------------------------------------------------------
# models and scenes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=6)
def _mesh(tris, seed=0):
    return wl.noisy_sphere(wl.segments_for_triangles(tris), seed=seed)


@functools.lru_cache(maxsize=2)
def _sbs(res):
    return wl.sbs_from_spheres(wl.spheres(64, seed=1), grid_res=res)


@functools.lru_cache(maxsize=2)
def _sbs_bytes(res):
    """_sbs with one byte per distance (the plain DX layout), four to a word."""
    hdr, nodes, vals, vf = _sbs(res)
    v = vf[vals.reshape(len(nodes), -1)[:, :11 ** 3]]
    dmax = math.sqrt(3.0) * 2.0 / (res // 8)
    q = np.zeros((len(nodes), 1332), np.uint8)
    q[:, :11 ** 3] = np.clip(np.rint((v + dmax) / (2 * dmax) * 255.0), 0, 255)
    hdr, nodes = hdr.copy(), nodes.copy()
    hdr["bytes_per_value"], hdr["aux_data"] = 1, SBS_LAYOUT_DX
    nodes["data_offset"] = np.arange(len(nodes)) * 333
    return hdr, nodes, q.reshape(-1).view(np.uint32), None


@functools.lru_cache(maxsize=2)
def _svs(lod):
    return wl.svs_from_spheres(wl.spheres(64, seed=1), lod)


@functools.lru_cache(maxsize=2)
def _octree(depth):
    return wl.frame_octree_from_spheres(wl.spheres(64, seed=1), depth)


@functools.lru_cache(maxsize=2)
def _scene(kind, size, depth=0):
    if kind == "svs":
        p = default_preset()
    else:
        p = parity_preset()
    sc = SceneRT(preset=p)
    if kind == "mesh":
        sc.AddInstance(sc.AddGeom_Triangles3f(*_mesh(size)), wl.IDENTITY)
    elif kind == "sbs":
        sc.AddInstance(sc.AddGeom_SdfSBS(*_sbs(size)), wl.IDENTITY)
    elif kind == "svs":
        sc.AddInstance(sc.AddGeom_SdfSVS(_svs(size)), wl.IDENTITY)
    elif kind == "instanced":  # three meshes and two octree models, `size` instances
        geoms = [sc.AddGeom_Triangles3f(*_mesh(n, n)) for n in (50000, 200000, 500000)]
        geoms += [sc.AddGeom_SdfFrameOctree(_octree(depth)) for _ in range(2)]
        for i, m in enumerate(wl.random_instances(size, seed=2)):
            sc.AddInstance(geoms[i % len(geoms)], m)
    elif kind == "mixed":  # a mesh, a brick set, a voxel set and an octree, `size` instances
        geoms = _four_kinds(sc)
        for i, m in enumerate(wl.random_instances(size, seed=7, scale=(0.3, 0.7), trans=1.4)):
            sc.AddInstance(geoms[i % 4], m)
    elif kind == "moving":
        geoms = [sc.AddGeom_Triangles3f(*_mesh(50000)), sc.AddGeom_SdfFrameOctree(_octree(6))]
        for i, m in enumerate(wl.random_instances(size, seed=5, scale=(0.1, 0.3), trans=2.5)):
            sc.AddInstance(geoms[i % 2], m)
    sc.CommitScene()
    return sc


def _four_kinds(sc):
    return [sc.AddGeom_Triangles3f(*_mesh(50000)), sc.AddGeom_SdfSBS(*_sbs_bytes(128)), sc.AddGeom_SdfSVS(_svs(6)),
            sc.AddGeom_SdfFrameOctree(_octree(6))]


def _camera(rng, radius, width, height):
    """One frame of a camera path: a fixed view moved by a few degrees."""
    az, el = 0.35 + math.radians(rng.uniform(-3, 3)), 0.25 + math.radians(rng.uniform(-2, 2))
    r = radius * (1 + rng.uniform(-0.02, 0.02))
    eye = (r * math.cos(el) * math.sin(az), r * math.sin(el), r * math.cos(el) * math.cos(az))
    return wl.camera(eye, width=width, height=height, tnear=TNEAR, tfar=TFAR)


def _query_rays(rng, n):
    """Unsorted rays from points on a radius-3 sphere towards points in the unit cube."""
    o = rng.normal(size=(n, 3))
    o *= 3.0 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(-0.9, 0.9, size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.empty((n, 8), np.float32)
    r[:, :3], r[:, 3], r[:, 4:7], r[:, 7] = o, TNEAR, d, TFAR
    return r


def _floats(n):
    return torch.empty(n, dtype=torch.float32, device="cuda")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _hits(h):
    """The hit records as their floating and whole parts (views of the buffer)."""
    h = h.view(-1, 8)
    return {"t": h[:, 0], "ids": h.view(torch.int32)[:, 1:4], "coords": h[:, 4:8]}


def _host_hits(h):
    return {"t": h["t"], "ids": np.stack([h["primId"], h["instId"], h["geomId"]], axis=-1).view(np.int32),
            "coords": h["coords"]}


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"case": case}
    if "scene" in case:
        st["scene"] = _scene(case["scene"], case["size"], case.get("depth", 0))
    if kind in ("query", "host_batch"):
        st["rays"] = _query_rays(rng, case.get("rays", 1))
    elif kind in ("frame", "host_frame"):
        w, h = case["width"], case["height"]
        st["rays"] = _floats(w * h * 8)
        st["scene"].generate_eye_rays(_camera(rng, 3.0, w, h), st["rays"].data_ptr(), _stream())
        if kind == "host_frame":
            st["rays"] = st["rays"].cpu().pin_memory()
            st["hits"] = torch.empty(w * h * 8, dtype=torch.float32).pin_memory()
        else:
            st["hits"] = _floats(w * h * 8)
    elif kind == "cameras":
        cams = wl.sphere_cameras(case["cameras"], radius=3.0, res_min=case["res_min"], res_max=case["res_max"], seed=3)
        views = wl.sphere_cameras(case["cameras"], radius=3.0, seed=seed, fixed_res=64)
        for c, v in zip(cams, views):  # sizes belong to the case, the directions to the seed
            c.world_view_inv[:] = v.world_view_inv[:]
            c.tfar = TFAR
        st["batch"] = CameraBatch(st["scene"], cams)
        st["hits"] = _floats(st["batch"].total_rays * 8)
    elif kind == "wavefront":
        n = case["side"] ** 2
        st["rays"], st["hits"], st["bounce"], st["bounce_hits"] = (_floats(n * 8) for _ in range(4))
        st["bounce"].zero_(), st["bounce_hits"].zero_()
        st["sky"] = torch.zeros(n, dtype=torch.float32, device="cuda")
        st["index"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        st["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        st["seed"] = int(rng.integers(1 << 30))
        st["scene"].generate_eye_rays(_camera(rng, 12.0, case["side"], case["side"]), st["rays"].data_ptr(), _stream())
    elif kind == "lambert_step":
        hdr, nodes, vals, vf = _sbs(case["size"])
        sc = SceneRT(preset=parity_preset())
        sc.AddInstance(sc.AddGeom_SdfSBS(hdr, nodes, vals, vf), wl.IDENTITY)
        sc.CommitScene()
        cams = wl.sphere_cameras(case["views"], radius=3.0, seed=seed, fixed_res=case["res"])
        n = case["views"] * case["res"] ** 2
        rays = _floats(n * 8)
        for k, c in enumerate(cams):
            c.tfar = TFAR
            sc.generate_eye_rays(c, rays.data_ptr() + k * case["res"] ** 2 * 32, _stream())
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        values = torch.from_numpy(vf).cuda()
        palette = 3 * 64
        values[palette:] += torch.randn(len(vf) - palette, generator=g, device="cuda") * (0.02 / case["size"])
        dimg = torch.randn(n, generator=g, device="cuda") / n
        st.update(scene=sc, rays=rays, values=values, dimage=dimg, image=_floats(n), grad=torch.zeros_like(values), n=n)
    elif kind == "render":
        w, h = case["width"], case["height"]
        mats = np.zeros(4, MATERIAL_DTYPE)
        mats["type"] = MATERIAL_COLORED
        mats["base_color"][:, :3] = rng.uniform(0.2, 1.0, (4, 3))
        mats["base_color"][:, 3] = (case["alpha"], 1.0, 1.0, 1.0)
        p = parity_preset()
        p.render_mode, p.spp = case["mode"], case["spp"]
        st.update(camera=_camera(rng, 4.0, w, h), lights=_lights(), preset=p, materials=mats,
                  image=torch.empty(w * h, dtype=torch.int32, device="cuda"))
    elif kind == "animate":
        w, h = case["width"], case["height"]
        st.update(camera=_camera(rng, 6.0, w, h), lights=_lights(),
                  poses=wl.random_instances(case["size"], seed=seed, scale=(0.1, 0.3), trans=2.5),
                  image=torch.empty(w * h, dtype=torch.int32, device="cuda"))
    elif kind == "load":
        w, h = case["width"], case["height"]
        st["mesh"] = wl.noisy_sphere(wl.segments_for_triangles(case["size"]), seed=int(seed))
        st["rays"] = torch.from_numpy(wl.eye_rays_host(_camera(rng, 3.0, w, h))).cuda()
        st["hits"] = _floats(w * h * 8)
    return st


def _lights():
    lights = np.zeros(3, LIGHT_DTYPE)
    lights[0] = ((0.577, 0.577, 0.577), LIGHT_DIRECT, (0.8, 0.8, 0.8), 0)
    lights[1] = ((1.0, 2.5, 2.0), LIGHT_POINT, (3.0, 3.0, 2.5), 0)
    lights[2] = ((0, 0, 0), LIGHT_AMBIENT, (0.1, 0.1, 0.1), 0)
    return lights


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case, sc = st["case"], st.get("scene")
    kind = case["kind"]
    if kind == "query":
        return _host_hits(sc.RayQuery_NearestHit(st["rays"][0, :4], st["rays"][0, 4:]))
    if kind == "host_batch":
        return _host_hits(sc.RayQuery_NearestHitBatch(st["rays"]))
    if kind == "frame":
        w, h = case["width"], case["height"]
        if case["order"] == "image":
            sc.trace_image(st["rays"].data_ptr(), st["hits"].data_ptr(), w, h, stream=_stream())
        else:
            sc.trace_device(st["rays"].data_ptr(), st["hits"].data_ptr(), w * h, stream=_stream())
        return _hits(st["hits"])
    if kind == "host_frame":
        sc.trace_host(st["rays"].data_ptr(), st["hits"].data_ptr(), case["width"] * case["height"])
        return _hits(st["hits"])
    if kind == "cameras":
        st["batch"].trace(st["hits"].data_ptr(), stream=_stream())
        return _hits(st["hits"])
    if kind == "wavefront":
        n, s = case["side"] ** 2, _stream()
        sc.trace_image(st["rays"].data_ptr(), st["hits"].data_ptr(), case["side"], case["side"], stream=s)
        sc.generate_bounce_rays_sorted(st["rays"].data_ptr(), st["hits"].data_ptr(), n, st["seed"],
                                       st["bounce"].data_ptr(), st["index"].data_ptr(), st["count"].data_ptr(),
                                       tnear=TNEAR, tfar=TFAR, stream=s)
        k = int(st["count"].item())  # the caller sizes the second wavefront by it
        sc.trace_device(st["bounce"].data_ptr(), st["bounce_hits"].data_ptr(), k, stream=s)
        # the open distance along each pixel's bounce, as an ambient-occlusion image takes it
        st["sky"].index_copy_(0, st["index"][:k].long(), st["bounce_hits"].view(-1, 8)[:k, 0])
        return {"primary": _hits(st["hits"]), "count": st["count"], "sky": st["sky"], "bounce_rays": st["bounce"],
                "bounce": _hits(st["bounce_hits"])}
    if kind == "lambert_step":
        s, n = _stream(), st["n"]
        size = (case["res"], case["res"] * case["views"])
        sc.update_sbs_values(st["values"].data_ptr(), st["values"].numel(), stream=s)
        sc.render_lambert(st["rays"].data_ptr(), n, wl.LIGHT, st["image"].data_ptr(), stream=s, image_size=size)
        st["grad"].zero_()
        sc.adjoint_lambert(st["rays"].data_ptr(), n, wl.LIGHT, st["dimage"].data_ptr(), st["grad"].data_ptr(),
                           stream=s, image_size=size)
        return {"image": st["image"], "grad": st["grad"]}
    if kind == "render":
        sc.SetPreset(st["preset"])
        sc.set_materials(st["materials"], [0, 1, 2, 3], [[0, 1], [1, 1], [2, 1], [3, 1]])
        sc.render_rgba8(st["camera"], st["lights"], BACKGROUND, st["image"].data_ptr(), stream=_stream())
        return st["image"]
    if kind == "animate":
        for i, m in enumerate(st["poses"]):
            sc.UpdateInstance(i, m, update_normal_matrix=True)
        sc.CommitScene()
        sc.render_rgba8(st["camera"], st["lights"], BACKGROUND, st["image"].data_ptr(), stream=_stream())
        return st["image"]
    # load
    sc = SceneRT(preset=parity_preset())
    sc.AddInstance(sc.AddGeom_Triangles3f(*st["mesh"], flags=BUILD_LOW), wl.IDENTITY)
    sc.CommitScene(BUILD_LOW)
    sc.trace_image(st["rays"].data_ptr(), st["hits"].data_ptr(), case["width"], case["height"], stream=_stream())
    st["scene"] = sc
    return _hits(st["hits"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Rays or cameras in, hits, pixels or gradients out, each once; a ray's
    operations are taken as 500 (a path of about ten node tests, a leaf and a
    hit point)."""
    kind = case["kind"]
    if kind in ("query", "host_batch"):
        rays = case.get("rays", 1)
        return {"bytes": 64 * rays, "flops": 500 * rays}
    if kind in ("frame", "host_frame"):
        rays = case["width"] * case["height"]
        return {"bytes": 64 * rays, "flops": 500 * rays}
    if kind == "cameras":
        cams = wl.sphere_cameras(case["cameras"], radius=3.0, res_min=case["res_min"], res_max=case["res_max"], seed=3)
        rays = sum(c.width * c.height for c in cams)
        return {"bytes": 32 * rays, "flops": 500 * rays}
    if kind == "wavefront":
        n = case["side"] ** 2
        k = int(0.3 * n * min(1.0, case["size"] / 1024))  # about three rays in ten hit 1024 instances
        return {"bytes": 64 * n + (32 + 32 + 4) * k, "flops": 500 * (n + k)}
    if kind == "lambert_step":
        n, bricks = case["views"] * case["res"] ** 2, 0.32 * case["size"] ** 2  # a surface's bricks
        values = bricks * 11 ** 3
        return {"bytes": 2 * 32 * n + 8 * n + 8 * values, "flops": 1500 * n}
    if kind == "render":
        rays = case["width"] * case["height"] * case["spp"]
        return {"bytes": 4 * case["width"] * case["height"], "flops": 1000 * rays}
    if kind == "animate":
        n = case["width"] * case["height"]
        return {"bytes": 4 * n + 256 * case["size"], "flops": 500 * n}
    tris, rays = case["size"], case["width"] * case["height"]
    return {"bytes": tris * (12 + 6 + 32) + 64 * rays, "flops": 100 * tris + 500 * rays}


def tolerance(case):
    if case["kind"] == "lambert_step":
        # gradients are float sums in the order that the atomics land: two runs differ by 6e-8 (2-norm), the
        # largest value by 5e-6; another rounding of the terms themselves adds a few units of 6e-8 to each
        return {"rel": 2e-6, "max": 2e-4}
    return "exact"  # hits and pixels are the reference's, bit for bit


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind not in ("query", "host_batch", "frame", "host_frame", "lambert_step", "load"):
        return None  # pixels are whole numbers; the others take too long without a traversal
    if kind == "load":
        rays = (case["width"] * case["height"])
        if rays * case["size"] > 2e10:
            return None
    st = prepare(case, seed)
    rays = torch.as_tensor(st["rays"]).reshape(-1, 8).cuda().double()
    if kind == "lambert_step":
        return _exact_lambert(case, st, rays)
    scene = case.get("scene", "mesh")
    if scene == "mesh":
        verts, tris = st["mesh"] if kind == "load" else _mesh(case["size"])
        if len(rays) * len(tris) > 4e10:
            return None
        t, coords = _nearest_triangle(rays, verts, tris)
    else:
        h = _march(rays, *(_sbs_grid(case["size"]) if scene == "sbs" else _svs_grid(case["size"])))
        t, coords = torch.where(h["hit"], h["t"], torch.full_like(h["t"], rays[0, 7].item())), None
    if kind == "query":
        return {"t": float(t[0]), "ids": None, "coords": None if coords is None else coords[0]}
    return {"t": t, "ids": None, "coords": coords}


def _encode(n):
    """Octahedral code of unit normals."""
    n = n / n.abs().sum(1, keepdim=True)
    p = n[:, :2]
    s = torch.where(p >= 0, 1.0, -1.0)
    return torch.where(n[:, 2:] <= 0, (1 - p.flip(1).abs()) * s, p)


def _nearest_triangle(rays, verts, tris):
    v = torch.from_numpy(verts).cuda().double()[torch.from_numpy(tris.astype(np.int64)).cuda()]
    A, E1, E2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = len(rays)
    best, uv = rays[:, 7].clone(), torch.zeros(n, 2, dtype=torch.float64, device="cuda")
    uv[:, 0] = 1.0
    which = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    step = max(1, min(len(A), (1 << 26) // n))
    o, d = rays[:, None, :3], rays[:, None, 4:7]
    for at in range(0, len(A), step):
        a, e1, e2 = A[None, at:at + step], E1[None, at:at + step], E2[None, at:at + step]
        p = torch.linalg.cross(d.expand(-1, a.shape[1], -1), e2.expand(n, -1, -1))
        tv = o - a
        q = torch.linalg.cross(tv, e1.expand(n, -1, -1))
        inv = 1.0 / (e1 * p).sum(-1)
        b = (tv * p).sum(-1) * inv
        c = (q * d).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        ok = (b >= -1e-6) & (c >= -1e-6) & (b + c <= 1 + 1e-6) & (t > rays[:, 3:4])
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        m, k = t.min(1)
        closer = m < best
        best = torch.where(closer, m, best)
        pick = torch.stack([c.gather(1, k[:, None])[:, 0], b.gather(1, k[:, None])[:, 0]], 1)
        uv = torch.where(closer[:, None], pick, uv)
        which = torch.where(closer, k + at, which)
    nrm = torch.linalg.cross(E1, E2)[which.clamp(min=0)]
    enc = _encode(nrm / nrm.norm(dim=1, keepdim=True))
    coords = torch.cat([uv, torch.where(which[:, None] >= 0, enc, torch.zeros_like(enc))], 1)
    return best, coords


def _grid_table(nodes, G):
    x, y = nodes["pos_xy"] >> 16, nodes["pos_xy"] & 0xFFFF
    z = nodes["pos_z_lod_size"] >> 16
    table = torch.full((G, G, G), -1, dtype=torch.int64, device="cuda")
    at = [torch.from_numpy(a.astype(np.int64)).cuda() for a in (x, y, z)]
    table[at[0], at[1], at[2]] = torch.arange(len(nodes), device="cuda")
    return table


def _sbs_grid(res, values=None):
    """Brick table, (bricks, 9, 9, 9) corner values, their indices, voxels per brick side, solver."""
    _, nodes, vals, vf = _sbs(res)
    idx = torch.from_numpy(vals.view(np.int32)).cuda().view(len(nodes), -1)[:, :11 ** 3].view(-1, 11, 11, 11)
    idx = idx[:, 1:10, 1:10, 1:10].contiguous()
    vf = torch.from_numpy(vf).cuda() if values is None else values
    return _grid_table(nodes, res // 8), vf[idx.long()], idx, 8, "march"


def _svs_grid(lod):
    nodes = _svs(lod)
    G = 1 << lod
    w = torch.from_numpy(nodes["values"].astype(np.int64)).cuda()
    q = torch.stack([(w[:, i // 4] >> (8 * (i % 4))) & 0xFF for i in range(8)], 1).double()
    dmax = 2 * 1.73205081 / G
    return _grid_table(nodes, G), (-dmax + 2 * dmax * q / 255).view(-1, 2, 2, 2), None, 1, "root"


def _trilinear(v, p):
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    a = v[:, 0:4] * (1 - x)[:, None] + v[:, 4:8] * x[:, None]
    b = a[:, 0:2] * (1 - y)[:, None] + a[:, 2:4] * y[:, None]
    return b[:, 0] * (1 - z) + b[:, 1] * z


def _march(rays, table, corners, idx, bs, solver):
    """Voxel march of every ray through the model's cube; in each voxel that
    holds the surface, sphere tracing ("march") or the first root of the field
    along the ray ("root").  Every loop pass moves each ray by one voxel or
    one tracing step."""
    dev, n = rays.device, len(rays)
    G, V = table.shape[0], corners.shape[1]
    N = G * bs
    size, eps = 2.0 / N, 1e-6
    o, d = rays[:, :3], rays[:, 4:7]
    inv = 1.0 / torch.where(d.abs() > 1e-36, d, torch.full_like(d, 1e-36))
    lo, hi = inv * (-1 - o), inv * (1 - o)
    t = torch.minimum(lo, hi).max(1).values.clamp(min=0.0)
    end = torch.maximum(lo, hi).min(1).values
    out = {"hit": torch.zeros(n, dtype=torch.bool, device=dev), "t": torch.zeros_like(t),
           "q": torch.zeros(n, 3, dtype=torch.float64, device=dev),
           "values": torch.zeros(n, 8, dtype=torch.float64, device=dev),
           "idx": torch.zeros(n, 8, dtype=torch.int64, device=dev),
           "early": torch.zeros(n, dtype=torch.bool, device=dev)}
    ray = torch.nonzero(t < end)[:, 0]  # the rays still under way, and their state
    t, end = t[ray], end[ray]
    tracing = torch.zeros(len(ray), dtype=torch.bool, device=dev)
    vals = torch.zeros(len(ray), 8, dtype=torch.float64, device=dev)
    vidx = torch.zeros(len(ray), 8, dtype=torch.int64, device=dev)
    q0 = torch.zeros(len(ray), 3, dtype=torch.float64, device=dev)
    near, far, s, steps = (torch.zeros(len(ray), dtype=torch.float64, device=dev) for _ in range(4))
    offs = torch.tensor([[(k >> 2) & 1, (k >> 1) & 1, k & 1] for k in range(8)], device=dev)
    flat = corners.reshape(-1)
    for _ in range(6000):
        if len(ray) == 0:
            break
        # 1. a voxel step for the rays that march
        m = torch.nonzero(~tracing & (t < end))[:, 0]
        if len(m):
            r, tm = ray[m], t[m]
            p = o[r] + (tm + 1e-9)[:, None] * d[r]
            cell = ((p + 1) / size).floor().long().clamp(0, N - 1)
            brick = cell // bs
            b = table[brick[:, 0], brick[:, 1], brick[:, 2]]
            in_brick = cell - brick * bs
            c = (in_brick[:, None, :] + offs)
            at = ((b.clamp(min=0)[:, None] * V + c[..., 0]) * V + c[..., 1]) * V + c[..., 2]
            v = flat[at].double()
            present = b >= 0
            surface = present & ((v.min(1).values <= 0) if solver == "march" else present)
            wide = ~present
            a_lo = torch.where(wide[:, None], brick * bs, cell).double() * size - 1
            a_hi = a_lo + torch.where(wide[:, None], float(bs), 1.0) * size
            x0, x1 = inv[r] * (a_lo - o[r]), inv[r] * (a_hi - o[r])
            tn, tf = torch.minimum(x0, x1).max(1).values, torch.maximum(x0, x1).min(1).values
            surface &= (tn > 0.01) & (tf > tn)
            go = torch.nonzero(surface)[:, 0]
            g = m[go]
            tracing[g] = True
            vals[g], near[g], far[g] = v[go], tn[go], tf[go]
            if idx is not None:
                vidx[g] = idx.view(-1)[at[go]].long()
            q0[g] = (o[r[go]] + tn[go][:, None] * d[r[go]] - a_lo[go]) / size
            s[g], steps[g] = 0.0, 0.0
            t[m] = torch.maximum(tf, tm) + 1e-9
        # 2. a tracing step for those inside a surface voxel
        m = torch.nonzero(tracing)[:, 0]
        if len(m):
            r, q_far = ray[m], (far[m] - near[m]) / size
            dist = _trilinear(vals[m], q0[m] + s[m][:, None] * d[r])
            if solver == "root":
                first = _first_root(vals[m], q0[m], d[r], q_far)
                early = dist <= eps
                hit = early | (first <= q_far)
                s[m] = torch.where(early, torch.zeros_like(first), first)
                stop = torch.ones_like(hit)
            else:
                early = (dist <= eps) & (steps[m] == 0)
                hit = (dist <= eps) & (s[m] <= q_far)
                stop = (dist <= eps) | (s[m] >= q_far) | (steps[m] >= 256)
            done = torch.nonzero(hit & stop)[:, 0]
            g, rd = m[done], r[done]
            out["hit"][rd], out["t"][rd] = True, near[g] + size * s[g]
            out["q"][rd], out["values"][rd] = q0[g] + s[g][:, None] * d[rd], vals[g]
            out["idx"][rd], out["early"][rd] = vidx[g], early[done]
            end[g] = -1.0
            tracing[m[stop]] = False
            cont = torch.nonzero(~stop)[:, 0]
            s[m[cont]] += dist[cont] / size
            steps[m[cont]] += 1
        keep = torch.nonzero(tracing | (t < end))[:, 0]
        if len(keep) < 0.9 * len(ray):
            ray, t, end, tracing, vals, vidx, q0, near, far, s, steps = (
                x[keep] for x in (ray, t, end, tracing, vals, vidx, q0, near, far, s, steps))
    return out


def _first_root(v, q0, d, q_far):
    """The first zero of the field on [0, q_far] (inf: none): a sign change among 32 pieces, bisected."""
    k = torch.linspace(0, 1, 33, dtype=torch.float64, device=v.device)
    f = torch.stack([_trilinear(v, q0 + (x * q_far)[:, None] * d) for x in k], 1)
    change = f[:, 1:] <= 0
    any_change = change.any(1)
    i = change.float().argmax(1)
    a, b = k[i] * q_far, k[i + 1] * q_far
    for _ in range(48):
        mid = 0.5 * (a + b)
        neg = _trilinear(v, q0 + mid[:, None] * d) <= 0
        a, b = torch.where(neg, a, mid), torch.where(neg, mid, b)
    return torch.where(any_change, b, torch.full_like(b, math.inf))


def _exact_lambert(case, st, rays):
    """Lambert image and its gradient with respect to the values, by the
    implicit function theorem at the hit point (a hit at a voxel's entry does
    not move with the values)."""
    h = _march(rays, *_sbs_grid(case["size"], st["values"]))
    image = torch.zeros(len(rays), dtype=torch.float64, device="cuda")
    grad = torch.zeros(len(st["values"]), dtype=torch.float64, device="cuda")
    L = torch.tensor(wl.LIGHT, dtype=torch.float32).double().cuda()
    r = torch.nonzero(h["hit"])[:, 0]
    v, p, d = h["values"][r], h["q"][r], rays[r, 4:7]
    e = 0.001
    shift = torch.eye(3, dtype=torch.float64, device="cuda") * e
    nrm = torch.stack([(_trilinear(v, p + shift[k]) - _trilinear(v, p - shift[k])) / (2 * e) for k in range(3)], 1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    shade = (nrm @ L).clamp(min=0)
    image[r] = shade
    lit = torch.nonzero(shade > 0)[:, 0]
    r, v, p, d, n = r[lit], v[lit], p[lit], d[lit], nrm[lit]
    bit = torch.tensor([[(k >> 2) & 1, (k >> 1) & 1, k & 1] for k in range(8)], device="cuda").double()
    w1 = bit[None] * p[:, None] + (1 - bit[None]) * (1 - p[:, None])  # (rays, 8, 3) weights per axis
    sg = 2 * bit[None] - 1
    dw = torch.stack([sg[..., 0] * w1[..., 1] * w1[..., 2], w1[..., 0] * sg[..., 1] * w1[..., 2],
                      w1[..., 0] * w1[..., 1] * sg[..., 2]], -1)
    g = (v[..., None] * dw).sum(1)
    n = g / g.norm(dim=1, keepdim=True)
    u = (L - (n @ L)[:, None] * n) / g.norm(dim=1, keepdim=True)
    hxy = (v * sg[..., 0] * sg[..., 1] * w1[..., 2]).sum(1)
    hxz = (v * sg[..., 0] * w1[..., 1] * sg[..., 2]).sum(1)
    hyz = (v * w1[..., 0] * sg[..., 1] * sg[..., 2]).sum(1)
    Hd = torch.stack([hxy * d[:, 1] + hxz * d[:, 2], hxy * d[:, 0] + hyz * d[:, 2], hxz * d[:, 0] + hyz * d[:, 1]], 1)
    gd = (g * d).sum(1)
    moves = torch.where(h["early"][r], torch.zeros_like(gd), (u * Hd).sum(1) / gd)
    dI = (u[:, None] * dw).sum(-1) - moves[:, None] * w1.prod(-1)
    grad.index_add_(0, h["idx"][r].reshape(-1), (st["dimage"].double()[r][:, None] * dI).reshape(-1))
    return {"image": image, "grad": grad}
