"""A recorded cull replayed after a batch of fewer objects on the same context. The batch is cut into finer
chunks than the recorded list, and the scratch the graph points into has to stay where it is. Equal to the
oracle before and after."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target, to_device
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu


# objects per resident warp (32 an SM): the list's chunk is the next multiple of 64, the batch's 64 to 256
@pytest.mark.parametrize("listed,batched", [(66, 62), (130, 60), (140, 120), (270, 250)])
def test_recorded_list_outlives_a_finer_batch(lib, listed, batched):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    sc = S.frustum_lod_scene(50_000, seed=3)
    rng = np.random.default_rng(9)
    v = view_for()
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        objs = np.ascontiguousarray(sc.objects[rng.integers(0, sc.count, warps * listed)])
        d, t = to_device(objs, "cuda"), Target.alloc(len(objs))
        n, recs, _ = O.cull(0, v, sc, objects=objs, threads=8)
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            c.draw_cull(v, t, objects=d, count=len(objs))
            c.capture_begin()
            c.draw_cull(v, t, objects=d, count=len(objs))
            g = c.capture_end()
            for k in range(2):
                t.commands.zero_()
                g.launch()
                side.synchronize()
                assert_records_equal(t.read(), (n, recs), f"replay {k}")
                if k == 0:
                    views, keep = (abi.BatchView * 2)(), []
                    for i, size in enumerate((warps * batched // 3, warps * batched - warps * batched // 3)):
                        part = np.ascontiguousarray(objs[:size])
                        pd, pt = to_device(part, "cuda"), Target.alloc(size)
                        views[i].view, views[i].mode = view_for(yaw=0.4 * i), 0
                        views[i].list, views[i].target = abi.RenderList(pd.data_ptr(), size), pt.ctype()
                        keep.append((part, pd, pt))
                    side.synchronize()
                    abi.check(c.lib.blz_cull_batch(c.ctx, views, 2, side.cuda_stream), "batch")
                    side.synchronize()
                    for i, (part, _, pt) in enumerate(keep):
                        bn, brecs, _ = O.cull(0, views[i].view, sc, objects=part, threads=8)
                        assert_records_equal(pt.read(), (bn, brecs), f"view {i}")
        assert c.check() == 0
