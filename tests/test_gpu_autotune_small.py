"""The batch autotuner on batches small enough for the default shape to cut its chunks finer: what it picks is no
slower than the default, which is one of its candidates, and the next small batch keeps its finer chunks."""
import ctypes as C

import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler
from tests.helpers import view_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,size", [(2, 4500), (16, 2000), (32, 60_000)])
def test_tuned_is_no_slower_than_the_default(lib, n, size, mixed):
    with Culler(0) as c:
        c.setup_for_rendering(S.frustum_lod_scene(60_000, seed=4))
        views, counts = (abi.BatchView * n)(), torch.zeros(n, dtype=torch.int32, device="cuda")
        commands = torch.zeros(n * size * 6, dtype=torch.int32, device="cuda")
        vis = torch.ones(size, dtype=torch.int32, device="cuda")
        for i in range(n):
            b = views[i]
            b.view, b.mode, b.visibility = view_for(yaw=0.3 * i), i % 2 if mixed else 0, vis.data_ptr()
            b.list = abi.RenderList(c.scene_tensors[0].data_ptr(), size)
            b.target = abi.CullTarget(commands.data_ptr() + i * size * 24, 24, size, counts.data_ptr() + 4 * i)

        def us():
            best, g = 1e9, C.c_void_p()
            abi.check(c.lib.blz_batch_graph_create(c.ctx, views, n, None, C.byref(g)), "graph")
            for _ in range(10):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(20):
                    abi.check(c.lib.blz_batch_graph_launch(g, None), "launch")
                b.record()
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b) * 50.0)
            abi.check(c.lib.blz_batch_graph_destroy(g), "destroy")
            return best

        default = us()
        best = abi.LaunchShape()
        abi.check(c.lib.blz_autotune_batch(c.ctx, views, n, 10, None, C.byref(best), None), "autotune")
        assert best.chunkObjects in (256, 512, 1024)
        tuned = us()
        assert tuned < 1.25 * default, (tuned, default, c.launch_shape())
