"""Lists short enough for one cluster of blocks (one launch): every pass, at the edges of warps, blocks, cluster
sizes and of the rule (4096 | 4097 objects), with a full and a short target. Bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300.culler import Culler, DevicePyramid, Target, to_device
from oracle import oracle as O
from tests.helpers import H, W, assert_records_equal, view_for
from tests.test_gpu_reject import rough_scene
from blitzen_gb300 import scenes as S

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 64, 65, 512, 513, 1025, 2049, 4096, 4097]


@pytest.fixture(scope="module")
def ctx(lib):
    c = Culler(0)
    sc = rough_scene(60)
    c.setup_for_rendering(sc)
    depth = O.depth_raster(view_for(), S.make_occluders(np.random.default_rng(8), 300, zmin=100.0, zmax=900.0), W, H)
    pyr = DevicePyramid(W, H)
    c.generate_depth_pyramid(pyr, torch.from_numpy(depth).cuda())
    yield c, sc, pyr, O.pyramid_build(depth)
    c.close()


@pytest.mark.parametrize("stride", [abi.STRIDE_VULKAN, abi.STRIDE_D3D12])
@pytest.mark.parametrize("mode", range(4))
@pytest.mark.parametrize("n", SIZES)
def test_short_list(ctx, n, mode, stride):
    c, sc, pyr, opyr = ctx
    rng = np.random.default_rng(n * 4 + mode)
    objs = np.ascontiguousarray(sc.objects[rng.choice(sc.count, n, replace=False)])
    vis0 = rng.integers(0, 3, n).astype(np.uint32)
    v = view_for(pw=float(pyr.desc.width), ph=float(pyr.desc.height))
    ovis = vis0.copy()
    cnt, recs, oflags = O.cull(mode, v, sc, objects=objs, vis=ovis, pyramid=opyr if mode >= 2 else None, stride=stride)
    dobjs = to_device(objs, "cuda")
    for capacity in (n, cnt // 2):
        vis = torch.from_numpy(vis0.view(np.int32).copy()).cuda()
        t = Target.alloc(n, stride)
        t.capacity = capacity
        before = c.launches
        if mode == 0:
            c.draw_cull(v, t, dobjs, n)
        elif mode == 1:
            c.draw_cull_first_pass(v, vis, t, dobjs, n)
        elif mode == 2:
            c.draw_cull_occlusion_pass(v, vis, pyr, t, dobjs, n)
        else:
            c.draw_cull_temporal(v, pyr, t, dobjs, n)
        assert c.launches - before == (1 if n <= 4096 else 2)
        assert c.flags() == oflags | (abi.FLAG_COMMAND_OVERFLOW if cnt > capacity else 0)
        stored = min(cnt, capacity)
        assert_records_equal(t.read(), (cnt, recs[:stored]), "records")
        assert not t.commands[stored * stride // 4:].any()  # nothing past the capacity or the count
        assert np.array_equal(vis.cpu().numpy().view(np.uint32), ovis)
