"""Threads with a context and a stream each, culling instanced over scenes of different LOD counts at the same time:
the shared memory one call asks of a kernel does not take away what the other's needs. Equal to the oracle."""
import threading

import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu

SLOTS = 900


@pytest.mark.parametrize("meshes", [(85, 250, 90, 240), (300, 900, 310, 890)], ids=str)
@pytest.mark.parametrize("recorded", [False, True])
def test_threads(lib, meshes, recorded):
    v, failed = view_for(zfar=1e4), []
    runs = []
    for k, m in enumerate(meshes):
        sc = S.frustum_lod_scene(4_000, seed=k, n_meshes=m, extent=500.0)
        c = Culler(0)
        c.setup_for_rendering(sc)
        ctr = O.new_counters(sc, SLOTS)
        cap = len(sc.lods) * SLOTS
        runs.append((c, sc, ctr, cap, torch.from_numpy(ctr.view(np.int32).reshape(-1).copy()).cuda(),
                     torch.full((cap,), -1, dtype=torch.int32, device="cuda"), Target.alloc(len(sc.lods)), torch.cuda.Stream()))
    torch.cuda.synchronize()
    gate = threading.Barrier(len(runs))

    def work(c, sc, ctr, cap, dctr, inst, t, stream):
        try:
            c.draw_instance_cull_pass(v, dctr, inst, SLOTS, t, stream=stream)
            gate.wait()
            for _ in range(2000):
                if recorded:
                    c.capture_begin(stream)
                c.draw_instance_cull_pass(v, dctr, inst, SLOTS, t, stream=stream)
                if recorded:
                    c.capture_end(stream).close()
        except Exception as e:  # noqa: BLE001 - reported by the test
            failed.append(e)

    threads = [threading.Thread(target=work, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == []
    for c, sc, ctr, cap, dctr, inst, t, _ in runs:
        assert c.check() == 0
        n, cmds, octr, oinst, _ = O.cull_instanced(v, sc, ctr, cap, SLOTS)
        assert_records_equal(t.read(), (n, cmds), "commands")
        assert np.array_equal(dctr.cpu().numpy().view(np.uint32), octr.view(np.uint32).reshape(-1))
        assert np.array_equal(inst.cpu().numpy().view(np.uint32), oinst)
        c.close()
