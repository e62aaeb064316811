"""The cluster emit launch with 1, 4 and 8 warps per tile: scenes on both sides of the lines between them (words of
visibility bits per tile, tiles), records and task form, full and short targets. Equal to the oracle word for
word; and a large scene of few clusters an object, whose tiles alone fill the chip, is not slowed down by more
warps than it has records for."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target, TaskTarget
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu
EYE = dict(position=(0.0, 0.0, -50.0))


def _check(c, sc, v, cap, tasks_cap, payload_cap):
    ids, t = torch.full((max(cap, 1),), -1, dtype=torch.int32, device="cuda"), Target.alloc(cap)
    c.cluster_cull(v, t, cluster_ids=ids)
    tt = TaskTarget.alloc(tasks_cap, payload_cap)
    c.cluster_task_cull(v, tt)
    c.flags()
    bound = O._cluster_upper_bound(sc, sc.objects)
    n, recs, oids, _ = O.cull_clusters(v, sc, capacity=bound, threads=8)
    m = min(n, cap)
    assert_records_equal(t.read(), (n, recs[:m]), "records")
    assert np.array_equal(ids.cpu().numpy().view(np.uint32)[:m], oids[:m])
    tasks, payloads = O.cluster_tasks(v, sc, threads=8)
    nt, np_, gt, gp = tt.read()
    assert (nt, np_) == (len(tasks), len(payloads))
    assert np.array_equal(gt, tasks[:tasks_cap]) and np.array_equal(gp, payloads[:payload_cap])
    return n, nt, np_


@pytest.mark.parametrize("n,per", [(1, 100), (33, 200), (2_000, 100), (12_345, 4), (12_345, 20), (25_600, 19), (25_600, 20), (25_601, 20),
                                   (25_600, 39), (25_600, 40), (25_601, 40), (50_000, 60), (150_000, 6)])
def test_forms(lib, n, per):
    sc = S.cluster_scene(n, seed=4, n_meshes=min(n, 24), clusters_per_mesh=per, extent=60.0 if n < 100 else 1000.0 * (n / 50_000) ** (1 / 3))
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        v = view_for(**EYE)
        k, nt, np_ = _check(c, sc, v, O._cluster_upper_bound(sc, sc.objects), sc.count, O._cluster_upper_bound(sc, sc.objects))
        _check(c, sc, v, k // 2, nt // 2, np_ // 2)


def test_time_of_many_objects_of_few_clusters(lib):
    """1M objects of up to 4 clusters, all in view. The test launch and the counting take about 130 us and the emit
    launch 48 with a warp per tile; with eight it took 327."""
    sc = S.cluster_scene(1_000_000, seed=3, n_meshes=24, clusters_per_mesh=4, extent=2700.0)
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        v, t = view_for(zfar=1e4, **EYE), Target.alloc(1_000_000)
        best = 1e9
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                c.cluster_cull(v, t)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 200.0)
        assert best < 300.0, best
