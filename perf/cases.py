"""The framework's measured work: ray-cast frames, batches, explicit rays, the
paged frame loop and octree builds, through the package's public entry points.

A case names an octree (``scene``: "icosphere", "terrain" or "menger"; the mesh
size ``size``, the octree ``depth``, the treelet ``levels``), what is done with
it (``kind``) and the sizes and options of that.  Scenes, cameras and resolutions
are the ranges of ``libsvo_b200.scenes``: octrees of depth 8 to 12, resolutions
from 64x64 to 3840x2160, fields of view from 25 to 60 degrees.  Every input is
made from the seed: the noise of the meshes, the voxel colours, the cameras, the
light, the explicit rays and the treelets that are paged.  A build keeps its mesh
and takes the vertex colours from the seed, so that its pool keeps its size.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libsvo_b200 as svo
from libsvo_b200.scenes import orbit_pose

# Floating-point operations of one step of a descent: the entry point (6), a
# child's slab (12) and the interval tests (4).
STEP_FLOPS = 22


def listed():
    ico9 = {"scene": "icosphere", "size": 5, "depth": 9, "levels": 4}
    ico10 = {"scene": "icosphere", "size": 5, "depth": 10, "levels": 5}
    ico11 = {"scene": "icosphere", "size": 6, "depth": 11, "levels": 6}
    ico12 = {"scene": "icosphere", "size": 6, "depth": 12, "levels": 6}
    return [
        # the smallest request of a rendering service: a thumbnail
        {"name": "frame_64", "kind": "frame", **ico9, "width": 64, "height": 64, "mode": 0},
        # one treelet holding a whole octree, the reference's simplest setting
        {"name": "frame_menger_512", "kind": "frame", "scene": "menger", "size": 5, "depth": 8, "levels": 0,
         "width": 512, "height": 512, "mode": 0},
        # a window of odd size, shaded by its normals, with the hit record of every
        # pixel (picking, depth compositing)
        {"name": "frame_hits_641x479", "kind": "frame", "scene": "terrain", "size": 257, "depth": 9, "levels": 4,
         "width": 641, "height": 479, "mode": 1, "hits": True},
        # the headline frame: a full HD view of the depth-11 octree
        {"name": "frame_1080p", "kind": "frame", **ico11, "width": 1920, "height": 1080, "mode": 0},
        # the same resolution over a flat breadth-first pool (the in-core raycaster)
        {"name": "frame_flat_1080p", "kind": "frame", **ico9, "width": 1920, "height": 1080, "mode": 0,
         "flat": True},
        # a viewer's frame: cast and copied to page-locked host memory, waited for
        {"name": "frame_host_720p", "kind": "host_frame", **ico10, "width": 1280, "height": 720, "mode": 0},
        # the largest frame: 4K with one shadow ray per hit, over a depth-12 octree
        {"name": "shadow_4k", "kind": "shadow", **ico12, "width": 3840, "height": 2160},
        # a million explicit rays without order (visibility queries, picking)
        {"name": "rays_1m", "kind": "rays", **ico11, "rays": 1000003},
        # a batch of views of uneven size over two octrees, one launch (offline
        # rendering of many views, a service's batch)
        {"name": "batch_48_views", "kind": "batch", "scene": "terrain", "size": 513, "depth": 10, "levels": 5,
         "views": 48, "min_side": 64, "max_side": 1024},
        # the out-of-core frame loop: treelets gone from the incore buffer are found
        # by the analysis pass, inserted and uploaded, and the frame is cast and shown
        {"name": "paged_1024", "kind": "paged", **ico10, "width": 1024, "height": 1024, "mode": 0,
         "treelets": 128},
        # octree builds from a mesh with vertex normals and colours: a small terrain,
        # and the depth-11 octree of the headline frame
        {"name": "build_terrain_d9", "kind": "build", "scene": "terrain", "size": 257, "depth": 9, "levels": 4},
        {"name": "build_icosphere_d11", "kind": "build", **ico11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "host_frame", "shadow", "shadow", "rays", "batch", "paged",
                       "build"])
    scene = rng.choice(["icosphere", "terrain"])
    depth = rng.randint(8, 11)
    if kind in ("paged", "host_frame"):
        depth = rng.randint(8, 10)
    size = rng.choice([4, 5, 6]) if scene == "icosphere" else rng.randint(100, 600)
    case = {"kind": kind, "scene": scene, "size": size, "depth": depth, "levels": rng.randint(3, 6)}
    if kind in ("frame", "host_frame", "shadow", "paged"):
        u = rng.random()
        case["width"] = max(16, int(64 * (2560 / 64) ** u) + rng.randint(-9, 9))
        case["height"] = max(16, int(64 * (1440 / 64) ** u) + rng.randint(-9, 9))
    if kind in ("frame", "host_frame", "paged"):
        case["mode"] = rng.choice([0, 0, 0, 0, 1, 3, 4, 5, 7])
    if kind == "frame":
        case["hits"] = rng.random() < 0.3
        if depth <= 9 and case["mode"] != 7 and rng.random() < 0.4:
            case["flat"] = True
    if kind == "rays":
        case["rays"] = _log_int(rng, 1000, 1500000)
    if kind == "batch":
        case["views"] = rng.randint(2, 64)
        case["min_side"] = rng.randint(33, 128)
        case["max_side"] = rng.randint(200, 1024)
    if kind == "paged":
        case["treelets"] = _log_int(rng, 8, 400)
    return case


# ---- inputs -----------------------------------------------------------------


def _mesh(case, seed):
    if case["scene"] == "icosphere":
        return svo.icosphere(case["size"], radius=0.4, octaves=3, amplitude=0.05, frequency=2.0, seed=seed)
    return svo.terrain(case["size"], octaves=6, base=-0.45, height=0.3, frequency=2.0, seed=seed)


def _host_scene(case, seed):
    if case["scene"] == "menger":
        return svo.Scene.menger(level=case["size"], depth=case["depth"], seed=seed)
    v, t = _mesh(case, seed)
    n, c = svo.vertex_attributes(v, t, seed)
    return svo.Scene.from_mesh(v, t, case["depth"], treelet_levels=case["levels"], normals=n, colors=c)


def _device_scene(case, seed):
    v, t = _mesh(case, seed)
    n, c = svo.vertex_attributes(v, t, seed)
    return svo.DeviceScene(v, t, case["depth"], treelet_levels=case["levels"], normals=n, colors=c)


def _resident(scene):
    i = scene.info
    mm = svo.TreeletMemoryManagerCuda(scene, i.num_treelets * i.treelet_bytes)
    mm.insertAll()
    mm.initDeviceBuffer()
    mm.sync()
    return mm


def _camera(scene, rng, width, height, headline=False):
    if scene == "terrain":  # an eye above the terrain, looking at a point on it
        eye = (rng.uniform(-0.45, 0.45), rng.uniform(0.0, 0.35), rng.uniform(-0.45, 0.45))
        target = (rng.uniform(-0.35, 0.35), -0.3, rng.uniform(-0.35, 0.35))
        return svo.Camera(eye, target, width, height, 60.0)
    if scene == "menger":
        return svo.orbit_camera(int(rng.integers(1 << 30)), width, height, radius=(1.5, 2.5), fov_deg=60.0)
    if headline:  # the orbit whose view the sphere fills
        return orbit_pose(2.5, rng.uniform(0, 360), rng.uniform(-30, 30), width, height, 25.0)
    return orbit_pose(rng.uniform(1.2, 2.5), rng.uniform(0, 360), rng.uniform(-40, 40), width, height,
                      rng.uniform(25, 60))


def _rays(rng, n):
    """Origins on the sphere of radius 1.2, directions to points of the cube."""
    o = rng.normal(size=(n, 3))
    o *= 1.2 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(-0.45, 0.45, size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (torch.from_numpy(o.astype(np.float32)).cuda(), torch.from_numpy(d.astype(np.float32)).cuda())


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    mesh_seed = 1 + seed % 100003
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "build":
        s["mesh"] = _mesh(case, case["size"])
        s["attributes"] = svo.vertex_attributes(*s["mesh"], mesh_seed)
        s["depth"], s["levels"] = case["depth"], case["levels"]
        return s

    # the octree, resident on the GPU
    s["cfg"] = svo.trace_cfg(stack_size=13)
    if kind in ("host_frame", "paged"):
        s["mm"] = _resident(_host_scene(case, mesh_seed))
    elif case.get("flat"):
        nodes, attribs = _host_scene(case, mesh_seed).flatten()
        s["hold"] = (torch.from_numpy(nodes.view(np.int32)).cuda(), torch.from_numpy(attribs.view(np.int32)).cuda())
        s["pool"] = (s["hold"][0], s["hold"][1], nodes.shape[0])
        s["cfg"] = svo.trace_cfg(svo.TRAVERSAL_FLAT, case["depth"])
    elif case["scene"] == "menger":
        s["hold"] = _resident(_host_scene(case, mesh_seed))
        s["pool"] = s["hold"].getDeviceIncoreBuffer()
    else:
        s["hold"] = _device_scene(case, mesh_seed)
        s["pool"] = s["hold"].buffers()

    if kind == "rays":
        s["origins"], s["dirs"] = _rays(rng, case["rays"])
        s["n"] = case["rays"]
        s["tsr"] = 2.0 * math.tan(math.radians(30.0)) / 1024.0  # a pixel of a 1024-line view
        s["hits"] = torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda")
        return s

    if kind == "batch":
        second = {"scene": "icosphere", "size": 5, "depth": 9, "levels": 4}
        s["hold2"] = _device_scene(second, mesh_seed)
        octrees = [svo.octree_desc(*s["pool"]), svo.octree_desc(*s["hold2"].buffers())]
        s["images"], views = [], []
        step = math.log(case["max_side"] / case["min_side"]) / case["views"]
        for k in range(case["views"]):  # the sides by turns from the whole range
            side = int(round(case["min_side"] * math.exp(step * ((k * 37 + 11) % case["views"] + 0.5))))
            cam = _camera(case["scene"] if k % 4 else second["scene"], rng, side, side)
            s["images"].append(torch.zeros((side, side), dtype=torch.int32, device="cuda"))
            views.append(svo.view_desc(cam.frame_params(), 0 if k % 4 else 1, s["images"][-1]))
        s["batcher"] = svo.Batcher(max_views=case["views"], max_octrees=2)
        s["batcher"].set(octrees, views, svo.batch_cfg(block_threads=128))
        return s

    w, h = case["width"], case["height"]
    s["params"] = _camera(case["scene"], rng, w, h, headline=w * h >= 1 << 20).frame_params(mode=case.get("mode", 0))
    on_host = kind in ("host_frame", "paged")
    s["image"] = torch.zeros((h, w), dtype=torch.int32, **({"pin_memory": True} if on_host else {"device": "cuda"}))
    if kind == "shadow":
        s["light"] = svo.shadow_cfg(svo.seeded_light(mesh_seed))
    if kind == "frame":
        s["hits"] = torch.zeros((h, w, 4), dtype=torch.int32, device="cuda") if case.get("hits") else None
    if kind == "paged":
        mm = s["mm"]
        mm.setUploadPolicy(svo.UPLOAD_PINNED)
        i = mm.info
        # treelets without sub-treelets: the last boundary level's, which the
        # builder numbers last
        gids = np.arange(i.num_treelets * 3 // 4, i.num_treelets)
        s["gone"] = sorted(int(g) for g in rng.choice(gids, size=min(case["treelets"], len(gids)), replace=False))
    return s


# ---- one pass ---------------------------------------------------------------


class _DeviceRecords:
    """A range of 8-byte records in device memory, for torch to look at."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count, 2), "typestr": "<i4", "data": (ptr, False), "version": 3}


def run(s):
    kind = s["kind"]
    if kind == "frame":
        svo.render(*s["pool"], s["params"], s["image"], s["hits"], cfg=s["cfg"])
        return s["image"] if s["hits"] is None else (s["image"], s["hits"])
    if kind == "host_frame":
        s["mm"].render_host(s["params"], s["image"], cfg=s["cfg"])
        return s["image"]
    if kind == "shadow":
        svo.render_shadow(*s["pool"], s["params"], s["image"], s["light"], cfg=s["cfg"])
        return s["image"]
    if kind == "rays":
        svo.trace_rays(s["pool"][0], s["pool"][2], s["origins"], s["dirs"], s["n"], s["tsr"], s["hits"], cfg=s["cfg"])
        return s["hits"]
    if kind == "batch":
        s["batcher"].launch()
        return s["images"]
    if kind == "paged":
        mm = s["mm"]
        for g in s["gone"]:
            mm.removeTreeletFromIncoreBuffer(g)
        mm.updateDeviceMemory()
        mm.performAnalysePass(s["params"])
        mm.render_host(s["params"], s["image"], cfg=s["cfg"])
        return s["image"]
    v, t = s["mesh"]
    n, c = s["attributes"]
    scene = svo.DeviceScene(v, t, s["depth"], treelet_levels=s["levels"], normals=n, colors=c)
    nodes, attribs, count = scene.buffers()
    return (torch.as_tensor(_DeviceRecords(scene, nodes, count), device="cuda"),
            torch.as_tensor(_DeviceRecords(scene, attribs, count), device="cuda"))


def exact(case, seed):
    """Every output is whole: pixels as bytes, records as words, a pool's records."""
    return None


# ---- what a pass cannot do without -------------------------------------------


def work(case):
    kind, depth = case["kind"], case["depth"]
    if kind == "build":
        # the voxels that the surface crosses, and a third as many inner nodes; a
        # record and an attribute written for each, the mesh read once
        leaves = 3.09 if case["scene"] == "icosphere" else 1.43
        nodes = 4.0 / 3.0 * leaves * 4.0 ** depth
        tris = 20 * 4 ** case["size"] if case["scene"] == "icosphere" else 2 * (case["size"] - 1) ** 2
        return {"bytes": 16 * nodes + 12 * tris + 18 * tris, "flops": 100 * nodes}
    if kind == "batch":  # the mean side^2 of a log-uniform side
        lo, hi = case["min_side"], case["max_side"]
        rays = case["views"] * (hi * hi - lo * lo) / (2 * math.log(hi / lo))
    elif kind == "rays":
        rays = case["rays"]
    else:
        rays = case["width"] * case["height"]
    # a ray: one descent to its leaf, the leaf's record and attribute, the pixel
    out = 24 + 16 if kind == "rays" else 4 + 16 * bool(case.get("hits"))
    b, f = rays * (16 + out), rays * depth * STEP_FLOPS
    if kind == "shadow":
        f *= 1.5
    if kind in ("host_frame", "paged"):
        b += 4 * rays
    if kind == "paged":  # the treelets' records and attributes, and a ray for 8x8 pixels
        b += case["treelets"] * 16 * 1.4 * 4.0 ** case["levels"]
        f += rays / 64 * depth * STEP_FLOPS
    return {"bytes": float(b), "flops": float(f)}
