"""The test that drops objects before the exact frustum test (surely_outside) never drops one the exact
test keeps: transforms with NaN, infinite, huge, tiny and negative values, quaternions of any length, bad
ids, and spheres within rounding of every plane. Records, counts, visibility and flags equal the oracle's,
in the one-call frame and in batches of every pass, with and without a surface table that fits on chip."""
import ctypes as C

import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, DevicePyramid, Target, to_device
from oracle import oracle as O
from tests.helpers import H, W, assert_records_equal, view_for

pytestmark = pytest.mark.gpu

VIEWS = [dict(), dict(position=(300.0, -200.0, 5000.0), yaw=2.1, pitch=0.4, zfar=700.0), dict(position=(1e6, 1e6, -1e6), yaw=-0.7, zfar=1e30)]


def rough_scene(meshes: int, n: int = 20_000, seed: int = 1) -> S.Scene:
    rng = np.random.default_rng(seed)
    surf, lods, _ = S.make_meshes(rng, meshes)
    objs, tr = S.make_objects(rng, n, 1000.0, meshes)
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e38, -1e38, 1e-38, 1e20, 1e-45, 3.0, -2.0], np.float32)
    rows = tr.view(np.float32).reshape(n, 8)
    k = rng.integers(0, n, n // 5)
    rows[k, rng.integers(0, 8, len(k))] = rng.choice(odd, len(k))
    k = rng.integers(0, n, n // 5)  # quaternions of any length
    rows[k, 4:] *= np.exp(rng.uniform(-6, 3, len(k))).astype(np.float32)[:, None]
    k = rng.integers(0, n, n // 10)
    rows[k, 3] *= -1.0
    surf["center"][: max(1, meshes // 8)] *= 200.0
    bad = rng.integers(0, n, 40)
    objs["transformId"][bad[:20]] = n + 5
    objs["surfaceId"][bad[20:]] = 0xFFFFFFF0
    if meshes > 4:
        surf["lodCount"][1] = 0xFFFFFFFF
    # spheres within a few ulp of the planes of the first view: a face's distance equal to the radius
    v = view_for()
    near = rng.integers(0, n, n // 4)
    z = rng.uniform(1.0, 900.0, len(near))
    face = rng.integers(0, 4, len(near))
    side = np.where(face < 2, 0, 1)
    a = np.where(side == 0, v.frustumLeft, v.frustumBottom).astype(np.float64)
    b = np.where(side == 0, v.frustumRight, v.frustumTop).astype(np.float64)
    sid = objs["surfaceId"][near]
    sid = np.where(sid < meshes, sid, 0)
    r = surf["radius"][sid].astype(np.float64) * rows[near, 3].astype(np.float64)
    x = (z * a + r) / b * (1.0 + rng.integers(-3, 4, len(near)) * 2.0 ** -24)
    rows[near, 0] = np.where(side == 0, np.where(face % 2, x, -x), 0.0)
    rows[near, 1] = np.where(side == 1, np.where(face % 2, x, -x), 0.0)
    rows[near, 2] = z
    surf["center"][meshes // 2:] = 0.0  # half of the meshes centred, so those spheres touch the planes
    return S.Scene(objs, tr, surf, lods, visibility=(rng.random(n) < 0.5).astype(np.uint32) * rng.integers(1, 4, n).astype(np.uint32))


@pytest.fixture(scope="module", params=[3, 60, 700], ids=lambda m: f"{m}_meshes")
def rough(request, lib):
    c = Culler(0)
    sc = rough_scene(request.param)
    c.setup_for_rendering(sc)
    depth = O.depth_raster(view_for(), S.make_occluders(np.random.default_rng(8), 300, zmin=100.0, zmax=900.0), W, H)
    yield c, sc, depth
    c.close()


@pytest.mark.parametrize("mode", [abi.HIZ_D3D12, abi.HIZ_VULKAN])
@pytest.mark.parametrize("k", range(len(VIEWS)))
def test_one_call_frame(rough, k, mode):
    c, sc, depth = rough
    opyr = O.pyramid_build(depth, mode)
    pyr = DevicePyramid(W, H, mode)
    v = view_for(pw=float(pyr.desc.width), ph=float(pyr.desc.height), **VIEWS[k])
    for ddepth in (torch.from_numpy(depth).cuda(), None):  # the pyramid built inside, then as it stands
        vis = torch.from_numpy(sc.visibility.view(np.int32).copy()).cuda()
        t1, t2 = Target.alloc(sc.count), Target.alloc(sc.count)
        c.cull_frame(v, vis, ddepth, pyr, t1, t2)
        flags = c.flags()
        ovis = sc.visibility.copy()
        n1, r1, f1 = O.cull(1, v, sc, vis=ovis)
        n2, r2, f2 = O.cull(2, v, sc, vis=ovis, pyramid=opyr)
        assert flags == f1 | f2
        assert_records_equal(t1.read(), (n1, r1), "pass 1")
        assert_records_equal(t2.read(), (n2, r2), "pass 2")
        assert np.array_equal(vis.cpu().numpy().view(np.uint32), ovis)


@pytest.mark.parametrize("modes", [(0,), (1,), (2,), (3,), (0, 1, 2, 3)], ids=str)
def test_batches(rough, modes):
    c, sc, depth = rough
    pyr, opyr = DevicePyramid(W, H), O.pyramid_build(depth)
    c.generate_depth_pyramid(pyr, torch.from_numpy(depth).cuda())
    n = 9
    views, keep = (abi.BatchView * n)(), []
    rng = np.random.default_rng(3)
    for i in range(n):
        size = int(rng.choice([1, 31, 513, 4000, sc.count]))
        objs = np.ascontiguousarray(sc.objects[np.sort(rng.choice(sc.count, size, replace=False))])
        vis = np.ascontiguousarray(rng.integers(0, 3, size).astype(np.uint32))
        d = (to_device(objs, "cuda"), torch.from_numpy(vis.view(np.int32).copy()).cuda(), Target.alloc(size))
        b = views[i]
        b.view, b.mode = view_for(**VIEWS[i % len(VIEWS)]), modes[i % len(modes)]
        b.list, b.visibility = abi.RenderList(d[0].data_ptr(), size), d[1].data_ptr()
        b.pyramid, b.target = C.pointer(pyr.desc), d[2].ctype()
        keep.append((objs, vis, d))
    abi.check(c.lib.blz_cull_batch(c.ctx, views, n, None), "batch")
    flags, expect = c.flags(), 0
    for i, (objs, vis, d) in enumerate(keep):
        ovis = vis.copy()
        m = modes[i % len(modes)]
        cnt, recs, f = O.cull(m, views[i].view, sc, objects=objs, vis=ovis, pyramid=opyr if m >= 2 else None)
        expect |= f
        assert_records_equal(d[2].read(), (cnt, recs), f"view {i} mode {m}")
        assert np.array_equal(d[1].cpu().numpy().view(np.uint32), ovis), f"view {i} mode {m}"
    assert flags == expect
