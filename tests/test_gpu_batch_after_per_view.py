"""Per-view launches and batches of one context in turn, with more chunks than resident warps: neither leaves
anything behind that makes the other skip chunks. Equal to the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target, to_device
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu


def test_batch_after_per_view(lib):
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    sc = S.frustum_lod_scene(50_000, seed=6)
    rng = np.random.default_rng(2)
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        sizes = [warps * 512 + 5000, 70_000, 300_000]  # the first alone has more chunks than there are warps
        views, keep = (abi.BatchView * 3)(), []
        for i, size in enumerate(sizes):
            objs = np.ascontiguousarray(sc.objects[rng.integers(0, sc.count, size)])
            d, t = to_device(objs, "cuda"), Target.alloc(size)
            views[i].view, views[i].mode = view_for(yaw=0.5 * i), 0
            views[i].list, views[i].target = abi.RenderList(d.data_ptr(), size), t.ctype()
            keep.append((d, t, O.cull(0, views[i].view, sc, objects=objs, threads=8)))
        for call in ("blz_cull_batch_per_view", "blz_cull_batch", "blz_cull_batch_per_view", "blz_cull_batch"):
            for _, t, _ in keep:
                t.commands.zero_()
            abi.check(getattr(c.lib, call)(c.ctx, views, 3, None), call)
            assert c.flags() == 0
            for i, (_, t, (n, recs, _)) in enumerate(keep):
                assert_records_equal(t.read(), (n, recs), f"{call} view {i}")
