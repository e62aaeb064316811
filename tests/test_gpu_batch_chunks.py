"""Batches around the sizes where the default shape's chunk changes (64, 128, 256, 512 objects), with uneven
views, called and as a batch graph. Equal to the oracle, word for word."""
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
N = 50_000


@pytest.fixture(scope="module")
def ctx(lib):
    c = Culler(0)
    sc = S.frustum_lod_scene(N, seed=5)
    c.setup_for_rendering(sc)
    depth = O.depth_raster(view_for(), S.make_occluders(np.random.default_rng(8), 300, zmin=100.0, zmax=900.0), W, H)
    pyr = DevicePyramid(W, H)
    c.generate_depth_pyramid(pyr, torch.from_numpy(depth).cuda())
    yield c, sc, pyr, O.pyramid_build(depth)
    c.close()


def make(ctx, total, modes, seed):
    """Three views of uneven size, `total` objects in all, drawn from the scene with repetition."""
    c, sc, pyr, _ = ctx
    rng = np.random.default_rng(seed)
    sizes = [total // 7, total // 100, total - total // 7 - total // 100]
    views, keep = (abi.BatchView * 3)(), []
    for i, size in enumerate(sizes):
        objs = np.ascontiguousarray(sc.objects[rng.integers(0, N, size)])
        vis = rng.integers(0, 2, size).astype(np.uint32)
        d = (to_device(objs, "cuda"), torch.from_numpy(vis.view(np.int32).copy()).cuda(), Target.alloc(size))
        b = views[i]
        b.view, b.mode = view_for(yaw=0.8 * i), modes[i % len(modes)]
        b.list, b.visibility = abi.RenderList(d[0].data_ptr(), size), d[1].data_ptr()
        b.pyramid, b.target = C.pointer(pyr.desc), d[2].ctype()
        keep.append((objs, vis, d))
    return views, keep


def check(ctx, views, keep):
    c, sc, _, opyr = ctx
    assert c.flags() == 0
    for i, (objs, vis, d) in enumerate(keep):
        ovis, m = vis.copy(), views[i].mode
        n, recs, _ = O.cull(m, views[i].view, sc, objects=objs, vis=ovis, pyramid=opyr if m >= 2 else None, threads=8)
        assert_records_equal(d[2].read(), (n, recs), f"view {i}")
        assert np.array_equal(d[1].cpu().numpy().view(np.uint32), ovis)


@pytest.mark.parametrize("modes", [(0,), (3,), (0, 1, 2)], ids=str)
@pytest.mark.parametrize("per_warp,more", [(1, 0), (64, 0), (64, 1), (128, 0), (128, 1), (256, 0), (256, 1)])
def test_chunk_edges(ctx, per_warp, more, modes):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    views, keep = make(ctx, warps * per_warp + more, modes, per_warp + more)
    abi.check(ctx[0].lib.blz_cull_batch(ctx[0].ctx, views, 3, None), "batch")
    check(ctx, views, keep)
    g = C.c_void_p()  # the same batch as a graph with its own scratch; pass 2 rewrites no word pass 2 left
    abi.check(ctx[0].lib.blz_batch_graph_create(ctx[0].ctx, views, 3, None, C.byref(g)), "graph")
    for _, vis, d in keep:
        d[1].copy_(torch.from_numpy(vis.view(np.int32)))
        d[2].commands.zero_()
    abi.check(ctx[0].lib.blz_batch_graph_launch(g, None), "launch")
    check(ctx, views, keep)
    abi.check(ctx[0].lib.blz_batch_graph_destroy(g), "destroy")
