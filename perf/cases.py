"""The calls a renderer makes of this framework, over the sizes it makes them at.

A case is one pass of one of these kinds, through `blitzen_gb300.culler.Culler` (batches through the
C entry point `blz_cull_batch`):

  dynamic    the dynamic objects of a scene rotated, written back and culled: a recorded frame, replayed
  frustum    frustum + LOD of one list, called directly (shadow and transparent lists have no occlusion)
  temporal   single-pass occlusion against the last frame's pyramid, called directly
  frame      a whole two-pass occlusion frame: "one_call" (depth known up front), "kept" (pass 1, pyramid,
             pass 2 over its survivors) or "passes" (the reference's three separate dispatches)
  instanced  per-LOD instance lists and one command per LOD
  clusters   object cull, then every cluster of the chosen LODs: "records" or "tasks", with or without Hi-Z
  depth      occluder boxes rasterised and the depth pyramid built from them
  batch      many views of uneven size over one resident scene, in one call

Cameras move a little from pass to pass, back and forth over a short path, so that the visibility
carried from frame to frame is the one a running renderer has: mostly stable, a few objects
appearing and disappearing. Scenes follow `blitzen_gb300.scenes`: positions uniform in a cube,
scale U[0.5, 2], random unit quaternions, occluder boxes in front of the camera.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, DevicePyramid, Target, TaskTarget

HIZ = {"d3d12": abi.HIZ_D3D12, "vulkan": abi.HIZ_VULKAN}
PATH = (0.0, 0.004, 0.008, 0.012, 0.008, 0.004)  # the camera's yaw (radians) over the frames of its path
SLOTS = 100_000                                   # instance slots per LOD of a large scene
IN_VIEW = 0.14                                    # share of a cube's objects inside a frustum at its centre
CLUSTER_IN_VIEW = 0.16                            # the same for a camera a little behind the centre


def listed() -> list[dict]:
    return [
        # the smallest call: a scene's 1,000 dynamic objects every frame, where launches are the cost
        dict(name="dynamic_1k", kind="dynamic", objects=1000, meshes=16, stride=24),
        # the plain frustum + LOD configuration: 100k objects, 16 meshes
        dict(name="frustum_100k", kind="frustum", objects=100_000, meshes=16, extent=1000.0, stride=24),
        # a small game scene, its whole frame in one call, ragged count, 720p
        dict(name="frame_50k", kind="frame", form="one_call", objects=50_021, meshes=40, extent=1200.0, stride=24,
             width=1280, height=720, hiz="d3d12"),
        # a mid-size scene in the renderer's own order (pass 1, its draws, pyramid, pass 2), Vulkan Hi-Z, 1440p
        dict(name="kept_400k", kind="frame", form="kept", objects=400_000, meshes=64, extent=2500.0, stride=24,
             width=2560, height=1440, hiz="vulkan"),
        # the reference's separate dispatches, D3D12 records, a window width that no vector load divides
        dict(name="passes_1m", kind="frame", form="passes", objects=1_000_003, meshes=300, extent=3000.0, stride=32,
             width=1366, height=768, hiz="d3d12"),
        # the stress frame: 4M objects, two-pass occlusion, 1080p
        dict(name="frame_4m", kind="frame", form="one_call", objects=4_000_000, meshes=64, extent=5000.0, stride=24,
             width=1920, height=1080, hiz="d3d12"),
        # instance lists of the stress scene: 64 meshes x 4 LODs
        dict(name="instanced_4m", kind="instanced", objects=4_000_000, meshes=64, extent=5000.0, stride=32),
        # instance lists of a scene with many different meshes: 500 x 4 LODs
        dict(name="instanced_2k_lods", kind="instanced", objects=250_000, meshes=500, extent=2000.0, stride=24),
        # meshlet culling behind occluders: 50k objects of about 200 clusters
        dict(name="clusters_50k", kind="clusters", form="records", objects=50_000, meshes=32, per_mesh=200, hiz="d3d12"),
        # the mesh-shader form without a pyramid (first frame, shadow views): most clusters survive to the cone test
        dict(name="tasks_12k", kind="clusters", form="tasks", objects=12_345, meshes=24, per_mesh=120, hiz=""),
        # occluder depth and its pyramid at 4K
        dict(name="depth_4k", kind="depth", boxes=2000, width=3840, height=2160, hiz="d3d12"),
        # 64 views (cameras, cascades) of 1k to 2M objects each over the 4M-object scene
        dict(name="batch_64", kind="batch", objects=4_000_000, meshes=64, views=64, low=1000, high=2_000_000,
             mode="temporal", width=1920, height=1080),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("dynamic", "frustum", "temporal", "frame", "frame", "instanced", "clusters", "depth", "batch"))
    width, height = rng.choice(((1280, 720), (1366, 768), (1600, 900), (1920, 1080), (2560, 1440), (1919, 1079)))
    hiz, stride = rng.choice(("d3d12", "vulkan")), rng.choice((24, 32))
    if kind == "dynamic":
        return dict(kind=kind, objects=_log(rng, 100, 20_000), meshes=rng.randint(1, 64), stride=stride)
    if kind == "depth":
        return dict(kind=kind, boxes=_log(rng, 50, 2000), width=width, height=height, hiz=hiz)
    if kind == "clusters":
        return dict(kind=kind, form=rng.choice(("records", "tasks")), objects=_log(rng, 500, 50_000),
                    meshes=rng.randint(4, 48), per_mesh=_log(rng, 20, 200), hiz=rng.choice(("", "d3d12", "vulkan")))
    if kind == "batch":
        return dict(kind=kind, objects=_log(rng, 200_000, 4_000_000), meshes=rng.randint(8, 128), views=rng.randint(2, 32),
                    low=_log(rng, 200, 2000), high=_log(rng, 20_000, 200_000), mode=rng.choice(("frustum", "temporal")),
                    width=width, height=height)
    n = _log(rng, 2000, 3_500_000)
    # extents as the configurations have them: about 100k objects in a cube of 2 km, 4M in one of 10 km
    base = dict(objects=n, meshes=_log(rng, 4, 500), extent=round(400.0 * (n / 5000) ** 0.36, 1), stride=stride)
    if kind == "frustum":
        return dict(kind=kind, **base)
    if kind == "instanced":
        return dict(kind=kind, **base)
    if kind == "temporal":
        return dict(kind=kind, **base, width=width, height=height, hiz=hiz)
    return dict(kind=kind, form=rng.choice(("one_call", "kept", "passes")), **base, width=width, height=height, hiz=hiz)


# ------------------------------------------------------------------ inputs

def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _tables(n: int, extent: float, meshes: int, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """Render objects and transforms with the distributions of scenes.make_objects, drawn on the GPU."""
    g = _generator(seed)
    f = torch.empty(n, 8, dtype=torch.float32, device="cuda")
    f[:, :3] = (torch.rand(n, 3, generator=g, device="cuda") * 2.0 - 1.0) * extent
    f[:, 3] = torch.rand(n, generator=g, device="cuda") * 1.5 + 0.5
    q = torch.randn(n, 4, generator=g, device="cuda", dtype=torch.float64)
    f[:, 4:] = (q / q.norm(dim=1, keepdim=True)).float()
    ids = torch.empty(n, 2, dtype=torch.int32, device="cuda")
    ids[:, 0] = torch.arange(n, device="cuda", dtype=torch.int32)
    ids[:, 1] = torch.randint(0, meshes, (n,), generator=g, device="cuda", dtype=torch.int32)
    objects = ids.cpu().numpy().view(abi.RENDER_OBJECT).reshape(n)
    transforms = f.cpu().numpy().view(abi.MESH_TRANSFORM).reshape(n)
    return objects, transforms


def _scene(case: dict, seed: int, extent: float, per_mesh: int = 0) -> S.Scene:
    rng = np.random.default_rng(seed)
    surfaces, lods, clusters = S.make_meshes(rng, case["meshes"], clusters_per_mesh=per_mesh)
    objects, transforms = _tables(case["objects"], extent, case["meshes"], seed)
    return S.Scene(objects, transforms, surfaces, lods, clusters=clusters)


def _pyramid_extent(width: int, height: int, hiz: str) -> tuple[float, float]:
    p, _ = abi.pyramid_layout(width, height, HIZ[hiz])
    return float(p.width), float(p.height)


def _view(width=1920, height=1080, hiz="d3d12", position=(0.0, 0.0, 0.0), yaw=0.0, pitch=0.0):
    pw, ph = _pyramid_extent(width, height, hiz)
    return abi.view_setup(S.fov_radians(), float(width), float(height), S.ZNEAR, S.STRESS_ZFAR, position, yaw, pitch, pw, ph)


def _path(width=1920, height=1080, hiz="d3d12", position=(0.0, 0.0, 0.0)):
    return [_view(width, height, hiz, position, yaw) for yaw in PATH]


def _boxes(seed: int, count: int, extent: float) -> np.ndarray:
    """Occluders in front of a camera at the origin, sized and spread as the stress scene's."""
    return S.make_occluders(np.random.default_rng(seed + 11), count, zmin=0.3 * extent, zmax=1.6 * extent,
                            size=(0.002 * extent, 0.04 * extent))


def _near_boxes(seed: int, count: int, extent: float) -> np.ndarray:
    """Fewer and larger ones, as the cluster scene's."""
    return S.make_occluders(np.random.default_rng(seed + 11), count, zmin=0.15 * extent, zmax=1.2 * extent,
                            size=(0.01 * extent, 0.2 * extent))


def _paint(boxes: np.ndarray, width: int, height: int, position=(0.0, 0.0, 0.0)) -> np.ndarray:
    """The reverse-Z depth of the boxes for a camera at `position` looking along +Z: each box's farthest
    corner over its screen rectangle, in float64."""
    focal = 1.0 / math.tan(S.fov_radians() / 2.0)
    p0, p5 = focal / (width / height), focal
    depth = np.zeros((height, width))
    corner = np.array([[(k >> a & 1) * 3 + a for a in range(3)] for k in range(8)])
    pts = boxes.astype(np.float64)[:, corner] - np.asarray(position)  # [box, corner, xyz]
    x, y, z = pts[..., 0], pts[..., 1], pts[..., 2]
    front = (z > S.ZNEAR).all(axis=1)
    sx, sy = ((x * p0 / z) * 0.5 + 0.5) * width, (0.5 - (y * p5 / z) * 0.5) * height
    x0, x1 = np.clip(np.floor(sx.min(1)), 0, width), np.clip(np.ceil(sx.max(1)), 0, width)
    y0, y1 = np.clip(np.floor(sy.min(1)), 0, height), np.clip(np.ceil(sy.max(1)), 0, height)
    d = S.ZNEAR / z.max(axis=1)
    for i in np.nonzero(front)[0]:
        part = depth[int(y0[i]):int(y1[i]), int(x0[i]):int(x1[i])]
        np.maximum(part, d[i], out=part)
    return depth


def _depth(case: dict, seed: int, extent: float) -> np.ndarray:
    return _paint(_boxes(seed, 2000, extent), case["width"], case["height"]).astype(np.float32)


def _upload(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


class State:
    """What a renderer keeps for one scene: the culler with its resident tables, the camera path and
    the output buffers."""

    def __init__(self, case: dict):
        self.case, self.frame, self.c = case, 0, Culler(torch.cuda.current_device())

    def next_view(self):
        v = self.path[self.frame % len(self.path)]
        self.frame += 1
        return v


# ------------------------------------------------------------------ prepare, by kind

def _prepare_dynamic(s: State, case: dict, seed: int) -> None:
    n = case["objects"]
    sc = _scene(case, seed, 300.0)
    s.c.setup_for_rendering(sc)
    s.table = s.c.scene_tensors[1].view(torch.float32).view(n, 8)
    s.ids = torch.arange(n, dtype=torch.int32, device="cuda")
    s.axes = _upload(_axes(seed, n))
    s.rotated = torch.zeros(n, 8, dtype=torch.float32, device="cuda")
    s.out = Target.alloc(n, case["stride"])
    start = s.table.clone()
    side = torch.cuda.Stream()

    def frame():
        s.c.rotate_transforms(s.ids, s.axes, ANGLE, s.rotated)
        s.c.update_object_transform_device(s.ids, s.rotated)
        s.c.draw_cull(_view(), s.out)

    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        frame()  # the unrecorded run that sizes the library's scratch
        s.c.capture_begin()
        frame()
        s.graph = s.c.capture_end()
        s.table.copy_(start)
    torch.cuda.current_stream().wait_stream(side)


ANGLE = 0.01


def _axes(seed: int, n: int) -> np.ndarray:
    a = np.random.default_rng(seed + 5).normal(size=(n, 3))
    return (a / np.linalg.norm(a, axis=1, keepdims=True)).astype(np.float32)


def _prepare_frustum(s: State, case: dict, seed: int) -> None:
    s.c.setup_for_rendering(_scene(case, seed, case["extent"]))
    s.path = _path()
    s.out = Target.alloc(case["objects"], case["stride"])


def _prepare_temporal(s: State, case: dict, seed: int) -> None:
    s.c.setup_for_rendering(_scene(case, seed, case["extent"]))
    s.path = _path(case["width"], case["height"], case["hiz"])
    s.pyramid = DevicePyramid(case["width"], case["height"], HIZ[case["hiz"]])
    s.c.generate_depth_pyramid(s.pyramid, _upload(_depth(case, seed, case["extent"])))
    s.out = Target.alloc(case["objects"], case["stride"])


def _prepare_frame(s: State, case: dict, seed: int) -> None:
    n = case["objects"]
    s.c.setup_for_rendering(_scene(case, seed, case["extent"]))
    s.path = _path(case["width"], case["height"], case["hiz"])
    s.depth = _upload(_depth(case, seed, case["extent"]))
    s.pyramid = DevicePyramid(case["width"], case["height"], HIZ[case["hiz"]])
    s.visibility = (torch.rand(n, generator=_generator(seed + 3), device="cuda") < 0.5).to(torch.int32)
    s.first, s.late = Target.alloc(n, case["stride"]), Target.alloc(n, case["stride"])


def _prepare_instanced(s: State, case: dict, seed: int) -> None:
    sc = _scene(case, seed, case["extent"])
    s.c.setup_for_rendering(sc)
    s.path = _path()
    n_lods = len(sc.lods)
    s.slots = min(SLOTS, case["objects"])
    if n_lods * s.slots > 30_000_000:  # many LODs: lists as long as a LOD's share of the scene can get
        s.slots = max(1024, 16 * case["objects"] // n_lods)
    counters = np.zeros(n_lods, abi.LOD_INSTANCE_COUNTER)
    counters["instanceOffset"] = np.arange(n_lods, dtype=np.uint64) * s.slots
    s.counters = _upload(counters.view(np.int32))
    s.instances = torch.zeros(n_lods * s.slots, dtype=torch.int32, device="cuda")
    s.out = Target.alloc(n_lods, case["stride"])


CLUSTER_EYE = (0.0, 0.0, -50.0)


def _prepare_clusters(s: State, case: dict, seed: int) -> None:
    n = case["objects"]
    extent = 1000.0 * (n / 50_000) ** (1 / 3)
    s.c.setup_for_rendering(_scene(case, seed, extent, per_mesh=case["per_mesh"]))
    hiz = case["hiz"] or "d3d12"
    s.path = _path(1920, 1080, hiz, CLUSTER_EYE)
    s.pyramid = None
    if case["hiz"]:
        s.pyramid = DevicePyramid(1920, 1080, HIZ[hiz])
        depth = _paint(_near_boxes(seed, 500, extent), 1920, 1080, CLUSTER_EYE)
        s.c.generate_depth_pyramid(s.pyramid, _upload(depth.astype(np.float32)))
    most = n * case["per_mesh"] // 4  # a quarter of the scene's clusters: more than a view draws
    if case["form"] == "tasks":
        s.out = TaskTarget.alloc(n, (most + 31) // 32 + n)
    else:
        s.out = Target.alloc(most, abi.STRIDE_VULKAN)
        s.cluster_ids = torch.zeros(most, dtype=torch.int32, device="cuda")


def _prepare_depth(s: State, case: dict, seed: int) -> None:
    s.boxes = _upload(_boxes(seed, case["boxes"], 5000.0).reshape(-1))
    s.view = _view(case["width"], case["height"], case["hiz"])
    s.depth = torch.zeros(case["height"], case["width"], dtype=torch.float32, device="cuda")
    s.pyramid = DevicePyramid(case["width"], case["height"], HIZ[case["hiz"]])


def _view_sizes(case: dict) -> list[int]:
    """The objects of each view, evenly spread between the smallest and the largest on a log scale."""
    low, high, views = case["low"], case["high"], case["views"]
    return [min(case["objects"], int(low * (high / low) ** ((k + 0.5) / views))) for k in range(views)]


def _prepare_batch(s: State, case: dict, seed: int) -> None:
    n, views = case["objects"], case["views"]
    extent = 5000.0 * (n / 4_000_000) ** (1 / 3)
    s.c.setup_for_rendering(_scene(case, seed, extent))
    rng, g = np.random.default_rng(seed + 17), _generator(seed + 19)
    resident = s.c.scene_tensors[0].view(n, 2)
    s.views = (abi.BatchView * views)()
    s.counts = torch.zeros(views, dtype=torch.int32, device="cuda")
    s.pyramids = []
    sizes = [int(x) for x in rng.permutation(_view_sizes(case))]
    # each view sees a random part of the scene, in the scene's order
    s.lists = [resident[torch.randperm(n, generator=g, device="cuda")[:k].sort().values].contiguous() for k in sizes]
    starts = np.concatenate([[0], np.cumsum([(x + 1) // 2 * 2 for x in sizes])])  # records start on 16 bytes
    s.commands = torch.zeros(int(starts[-1]) * 6 + 4, dtype=torch.int32, device="cuda")
    w, h = case["width"], case["height"]
    for k in range(views):
        at = tuple(float(x) for x in rng.uniform(-extent, extent, 3).astype(np.float32))
        v = _view(w, h, "d3d12", at, float(rng.uniform(-math.pi, math.pi)), float(rng.uniform(-0.5, 0.5)))
        b = s.views[k]
        b.view, b.list = v, abi.RenderList(s.lists[k].data_ptr(), sizes[k])
        b.mode = abi.MODE_TEMPORAL if case["mode"] == "temporal" else abi.MODE_FRUSTUM
        b.target = abi.CullTarget(s.commands.data_ptr() + int(starts[k]) * 24, 24, sizes[k], s.counts.data_ptr() + 4 * k)
        if case["mode"] == "temporal":
            depth = torch.zeros(h, w, dtype=torch.float32, device="cuda")
            m = np.frombuffer(bytes(v.viewMatrix), np.float32).reshape(4, 4)[:3, :3].astype(np.float64)
            box = _boxes(seed + k, 2000, extent).astype(np.float64).reshape(-1, 2, 3) @ m.T + np.asarray(at)
            box = np.concatenate([box.min(axis=1), box.max(axis=1)], axis=1).astype(np.float32)
            s.c.raster_boxes(v, _upload(box.reshape(-1)), depth, w, h)
            s.pyramids.append(DevicePyramid(w, h, abi.HIZ_D3D12))
            s.c.generate_depth_pyramid(s.pyramids[-1], depth)
            b.pyramid = C.pointer(s.pyramids[-1].desc)
    s.lib = abi.load()


def prepare(case: dict, seed: int) -> State:
    s = State(case)
    globals()["_prepare_" + case["kind"]](s, case, seed)
    return s


# ------------------------------------------------------------------ run

def run(s: State):
    case, c = s.case, s.c
    kind = case["kind"]
    if kind == "dynamic":
        s.graph.launch()
        return {"transforms": s.table, "count": s.out.count, "commands": s.out.commands}
    if kind == "frustum":
        c.draw_cull(s.next_view(), s.out)
        return {"count": s.out.count, "commands": s.out.commands}
    if kind == "temporal":
        c.draw_cull_temporal(s.next_view(), s.pyramid, s.out)
        return {"count": s.out.count, "commands": s.out.commands}
    if kind == "frame":
        view = s.next_view()
        if case["form"] == "one_call":
            c.cull_frame(view, s.visibility, s.depth, s.pyramid, s.first, s.late)
        elif case["form"] == "kept":
            c.frame_first_pass(view, s.visibility, s.first)
            c.generate_depth_pyramid(s.pyramid, s.depth)
            c.frame_occlusion_pass(s.pyramid, s.late)
        else:
            c.draw_cull_first_pass(view, s.visibility, s.first)
            c.generate_depth_pyramid(s.pyramid, s.depth)
            c.draw_cull_occlusion_pass(view, s.visibility, s.pyramid, s.late)
        return {"pyramid": s.pyramid.storage, "visibility": s.visibility, "count1": s.first.count,
                "commands1": s.first.commands, "count2": s.late.count, "commands2": s.late.commands}
    if kind == "instanced":
        c.draw_instance_cull_pass(s.next_view(), s.counters, s.instances, s.slots, s.out)
        return {"counters": s.counters, "instances": s.instances, "count": s.out.count, "commands": s.out.commands}
    if kind == "clusters":
        if case["form"] == "tasks":
            c.cluster_task_cull(s.next_view(), s.out, pyramid=s.pyramid)
            return {"counts": s.out.counts, "tasks": s.out.tasks, "payloads": s.out.payloads}
        c.cluster_cull(s.next_view(), s.out, pyramid=s.pyramid, cluster_ids=s.cluster_ids)
        return {"count": s.out.count, "commands": s.out.commands, "cluster_ids": s.cluster_ids}
    if kind == "depth":
        c.raster_boxes(s.view, s.boxes, s.depth, case["width"], case["height"])
        c.generate_depth_pyramid(s.pyramid, s.depth)
        return {"depth": s.depth, "pyramid": s.pyramid.storage}
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    abi.check(s.lib.blz_cull_batch(c.ctx, s.views, case["views"], stream), "blz_cull_batch")
    return {"counts": s.counts, "commands": s.commands}


# ------------------------------------------------------------------ what a pass cannot do without

def _pyramid_texels(width: int, height: int, hiz: str) -> int:
    return abi.pyramid_layout(width, height, HIZ[hiz])[1] // 4


def work(case: dict) -> dict:
    """Each table row, depth texel and visibility word of the pass read once and each record, list entry
    and texel written once; operations of the tests in the shaders' own arithmetic (a frustum test 75, a
    sphere projection with its Hi-Z test and LOD selection 70)."""
    kind, n = case["kind"], case.get("objects", 0)
    stride = case.get("stride", 24)
    seen = IN_VIEW * n
    if kind == "dynamic":
        return {"bytes": n * (4 + 12 + 32 + 32 + 8) + seen * stride + 4, "flops": n * 115 + seen * 25}
    if kind == "frustum":
        return {"bytes": n * 40 + seen * stride + 4, "flops": n * 75 + seen * 25}
    if kind == "temporal":
        return {"bytes": n * 40 + seen / 2 * stride + 4, "flops": n * 75 + seen * 70}
    if kind == "frame":
        texels = _pyramid_texels(case["width"], case["height"], case["hiz"])
        image = case["width"] * case["height"] * 4 + texels * 4
        return {"bytes": n * 44 + seen / 2 * stride + image + 8, "flops": n * 75 + seen * 70 + texels * 3}
    if kind == "instanced":
        return {"bytes": n * 40 + seen * 4 + case["meshes"] * 4 * (32 + 16 + stride), "flops": n * 75 + seen * 25}
    if kind == "clusters":
        tested = CLUSTER_IN_VIEW * n * case["per_mesh"]
        kept = tested * (0.02 if case["hiz"] else 0.5)
        per = 28 if case["form"] == "records" else 4
        return {"bytes": n * 40 + case["meshes"] * case["per_mesh"] * 32 + kept * per,
                "flops": n * 75 + tested * (75 + (70 if case["hiz"] else 45))}
    if kind == "depth":
        texels = _pyramid_texels(case["width"], case["height"], case["hiz"])
        return {"bytes": case["boxes"] * 24 + case["width"] * case["height"] * 4 + texels * 4, "flops": texels * 3}
    tests = sum(_view_sizes(case))
    hiz = case["mode"] == "temporal"
    # every list once, and of the shared transforms each row that some view needs, once
    rows = n * (1.0 - math.exp(-tests / n))
    return {"bytes": tests * 8 + rows * 32 + tests * 0.1 * 24, "flops": tests * 75 + tests * 0.1 * (70 if hiz else 25)}


# ------------------------------------------------------------------ the computed numbers in 64 bits

def _min_levels(depth: np.ndarray, width: int, height: int, hiz: str) -> np.ndarray:
    """Every mip of the depth's pyramid, mips back to back, from the two sampling rules: the minimum of
    the 2x2 texels below (absent ones count as 0), or of the bilinear footprint clamped to the edge."""
    def two_by_two(a, w, h):
        out = np.zeros((2 * h, 2 * w))
        part = a[:2 * h, :2 * w]
        out[:part.shape[0], :part.shape[1]] = part
        return out.reshape(h, 2, w, 2).min(axis=(1, 3))

    def footprint(a, w, h):
        def ends(size, source):
            u = (np.arange(size) + 0.5) / size * source - 0.5
            lo = np.floor(u)
            hi = lo + (u > lo)
            return np.clip(lo, 0, source - 1).astype(int), np.clip(hi, 0, source - 1).astype(int)
        x0, x1 = ends(w, a.shape[1])
        y0, y1 = ends(h, a.shape[0])
        rows = np.minimum(a[y0], a[y1])
        return np.minimum(rows[:, x0], rows[:, x1])

    level = two_by_two if hiz == "d3d12" else footprint
    w, h = width // 2, height // 2
    if hiz == "vulkan":
        w, h = (1 << (v - 1).bit_length() - 1 for v in (width, height))
    out, a = [], depth.astype(np.float64)
    for _ in range(max(w, h).bit_length() - 1):
        a = level(a, w, h)
        out.append(a.reshape(-1))
        w, h = max(1, w // 2), max(1, h // 2)
    return np.concatenate(out)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "dynamic":
        _, transforms = _tables(case["objects"], 300.0, case["meshes"], seed)
        t = transforms.view(np.float32).reshape(-1, 8).astype(np.float64)
        half = np.float64(np.float32(ANGLE)) * 0.5
        r, w = math.sin(half) * _axes(seed, len(t)).astype(np.float64), math.cos(half)
        q, qw = t[:, 4:7], t[:, 7:8]
        t = np.concatenate([t[:, :4], w * q + r * qw + np.cross(r, q), w * qw - (r * q).sum(axis=1, keepdims=True)], axis=1)
        return {"transforms": t, "count": None, "commands": None}
    if kind == "frame":
        depth = _depth(case, seed, case["extent"])
        return {"pyramid": _min_levels(depth, case["width"], case["height"], case["hiz"]), "visibility": None, "count1": None,
                "commands1": None, "count2": None, "commands2": None}
    if kind == "depth":
        depth = _paint(_boxes(seed, case["boxes"], 5000.0), case["width"], case["height"])
        return {"depth": depth, "pyramid": _min_levels(depth, case["width"], case["height"], case["hiz"])}
    return None
