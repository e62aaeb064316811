"""Batches of many small views, and of views around the 256 chunks a scanning warp takes a round: each view's
records, count and overflow equal the oracle's, and the call's time grows with the views no faster than the
work that a view cannot do without."""
import ctypes as C

import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, to_device
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu
N = 20_000


class Batch:
    def __init__(self, c, sc, sizes, capacity=None, seed=0):
        self.c, self.sc, n = c, sc, len(sizes)
        self.objs = np.ascontiguousarray(sc.objects[np.random.default_rng(seed).integers(0, sc.count, max(sizes + [1]))])
        self.dobjs = to_device(self.objs, "cuda")
        self.counts = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        self.capacity = [s if capacity is None else min(s, capacity) for s in sizes]
        self.start = np.concatenate([[0], np.cumsum([(x + 1) // 2 * 2 for x in self.capacity])])
        self.commands = torch.zeros(int(self.start[-1]) * 6 + 4, dtype=torch.int32, device="cuda")
        self.views, self.sizes = (abi.BatchView * n)(), sizes
        for i, size in enumerate(sizes):
            b = self.views[i]
            b.view, b.mode, b.list = view_for(yaw=0.1 * i), 0, abi.RenderList(self.dobjs.data_ptr(), size)
            b.target = abi.CullTarget(self.commands.data_ptr() + 24 * int(self.start[i]), 24, self.capacity[i], self.counts.data_ptr() + 4 * i)

    def run(self):
        abi.check(self.c.lib.blz_cull_batch(self.c.ctx, self.views, len(self.sizes), None), "batch")

    def check(self, which):
        counts, words = self.counts.cpu().numpy(), self.commands.cpu().numpy().view(np.uint32)
        for i in which:
            if self.sizes[i] == 0:
                assert counts[i] == 0
                continue
            n, recs, _ = O.cull(0, self.views[i].view, self.sc, objects=self.objs[:self.sizes[i]], threads=8)
            m = min(n, self.capacity[i])
            at = int(self.start[i]) * 6
            assert counts[i] == n
            assert_records_equal((n, words[at:at + 6 * m].reshape(m, 6)), (n, recs[:m]), f"view {i}")


@pytest.mark.parametrize("sizes", [[1] * 3, [40] * 700, [0, 50, 0] * 300, [64 * 255] + [1] * 20, [64 * 256, 1], [64 * 256 + 1, 3], [64 * 257] * 3,
                                   [300_000] * 2, [200_000] + [10] * 4000], ids=lambda s: f"{len(s)}x{max(s)}")
def test_views(lib, sizes):
    sc = S.frustum_lod_scene(N, seed=5)
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        b = Batch(c, sc, sizes)
        b.run()
        assert c.flags() == 0
        k = len(b.sizes)
        b.check(sorted({0, 1 % k, k // 2, k - 1}))
        short = Batch(c, sc, b.sizes, capacity=2)
        short.run()
        over = any((short.counts.cpu().numpy() > np.array(short.capacity)))
        assert c.flags() == (abi.FLAG_COMMAND_OVERFLOW if over else 0)
        short.check(sorted({0, k // 2, k - 1}))


def test_time_of_many_views(lib):
    """10,000 views of 50 objects, replayed, against 1,024 of them: the decide launch takes twice as long and nothing
    else does, so the call takes less than three times (a block scanning each view's one chunk: 4.1 times)."""
    sc = S.frustum_lod_scene(N, seed=5)
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        us = []
        for n in (1024, 10_000):
            b, g = Batch(c, sc, [50] * n), C.c_void_p()
            abi.check(c.lib.blz_batch_graph_create(c.ctx, b.views, n, None, C.byref(g)), "graph")
            best = 1e9
            for _ in range(10):
                s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                s.record()
                for _ in range(20):
                    abi.check(c.lib.blz_batch_graph_launch(g, None), "launch")
                e.record()
                torch.cuda.synchronize()
                best = min(best, s.elapsed_time(e) * 50.0)
            us.append(best)
            abi.check(c.lib.blz_batch_graph_destroy(g), "destroy")
        assert us[1] < 3.0 * us[0], us
