"""Batches decided in the order of their chunks' places in their views (a transform table of 48 MiB or more, 2M objects
or more, up to 256 views): called and as a graph, on both sides of each limit, with empty and one-chunk views between
long ones, and with views of 2^15 chunks and more, whose ranks take 64 bits. Equal to the oracle."""
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
N = (48 << 20) // 32  # the smallest table that is ordered for
M2 = 1 << 21          # objects, in chunks of 512


@pytest.fixture(scope="module")
def ctx(lib):
    c, sc = Culler(0), S.frustum_lod_scene(N, seed=5, extent=2000.0)
    c.setup_for_rendering(sc)
    objs = np.ascontiguousarray(sc.objects[np.random.default_rng(1).integers(0, N, (1 << 15) * 256 + 700)])
    yield c, sc, objs, to_device(objs, "cuda"), {}
    c.close()


def _reference(ctx, size, k):
    c, sc, objs, _, cache = ctx
    if (size, k) not in cache:
        n, recs, _ = O.cull(0, view_for(yaw=0.7 * k, zfar=1e4), sc, objects=objs[:size], threads=O.default_threads())
        cache[size, k] = n, recs
    return cache[size, k]


def _run(ctx, sizes, chunk, graph):
    c, sc, objs, dobjs, _ = ctx
    n = len(sizes)
    start = np.concatenate([[0], np.cumsum([(s // 2 + 2) // 2 * 2 for s in sizes])])  # half of a list is room enough for a view's
    counts = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    commands = torch.zeros(int(start[-1]) * 6 + 4, dtype=torch.int32, device="cuda")
    views = (abi.BatchView * n)()
    for i, size in enumerate(sizes):
        b = views[i]
        b.view, b.mode, b.list = view_for(yaw=0.7 * (i % 3), zfar=1e4), 0, abi.RenderList(dobjs.data_ptr(), size)
        b.target = abi.CullTarget(commands.data_ptr() + 24 * int(start[i]), 24, int(start[i + 1] - start[i]), counts.data_ptr() + 4 * i)
    c.set_launch_shape(256, 2, 0, chunk)
    before = c.launches
    if graph:
        g = C.c_void_p()
        abi.check(c.lib.blz_batch_graph_create(c.ctx, views, n, None, C.byref(g)), "create")
        for _ in range(2):
            abi.check(c.lib.blz_batch_graph_launch(g, None), "launch")
        abi.check(c.lib.blz_batch_graph_destroy(g), "destroy")
    else:
        abi.check(c.lib.blz_cull_batch(c.ctx, views, n, None), "batch")
    launches = c.launches - before
    assert c.check() == 0
    got, words = counts.cpu().numpy(), commands.cpu().numpy().view(np.uint32)
    for i, size in enumerate(sizes):
        m, recs = _reference(ctx, size, i % 3)
        at = int(start[i]) * 6
        assert_records_equal((int(got[i]), words[at:at + 6 * m].reshape(m, 6)), (m, recs), f"view {i}")
    c.set_launch_shape(256, 2)
    return launches


@pytest.mark.parametrize("graph", [False, True], ids=["call", "graph"])
@pytest.mark.parametrize("sizes", [[M2 - 512, 512], [M2 - 1024, 512], [1_500_000, 0, 3, 600_000, 0, 70_001], [8192] * 256, [8192] * 257,
                                   [M2]], ids=lambda s: f"{len(s)}x{s[0]}")
def test_limits(ctx, sizes, graph):
    launches = _run(ctx, sizes, 512, graph)
    if not graph:  # decide, scan, scatter, and the order where the rule has it
        chunks = sum(max(1, (s + 511) // 512) for s in sizes)
        assert launches == (4 if 1 < len(sizes) <= 256 and chunks * 512 >= M2 else 3)


@pytest.mark.parametrize("graph", [False, True], ids=["call", "graph"])
@pytest.mark.parametrize("more", [-256, 0, 700])
def test_views_of_many_chunks(ctx, more, graph):
    _run(ctx, [(1 << 15) * 256 + more, 40_000, 1, 1_000_000], 256, graph)
