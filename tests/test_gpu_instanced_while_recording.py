"""A direct instanced cull of many LODs whose scratch has to grow while another context's frame is being
recorded, by the same thread or another: the recording stays valid, and both results equal the oracle's."""
import threading

import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu

SLOTS = 2_000


@pytest.mark.parametrize("threaded", [False, True])
def test_growth_leaves_a_recording_alone(lib, threaded):
    many = S.frustum_lod_scene(700_000, seed=5, n_meshes=300, extent=3000.0)
    small = S.frustum_lod_scene(20_000, seed=6)
    v = view_for()
    with Culler(0) as rec, Culler(0) as c:
        rec.setup_for_rendering(small)
        c.setup_for_rendering(many)
        cap = len(many.lods) * SLOTS
        ctr = O.new_counters(many, SLOTS)
        dctr = torch.from_numpy(ctr.view(np.int32).reshape(-1).copy()).cuda()
        inst = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
        t, rt = Target.alloc(len(many.lods)), Target.alloc(small.count)
        a, b = torch.cuda.Stream(), torch.cuda.Stream()

        def direct():
            c.draw_instance_cull_pass(v, dctr, inst, SLOTS, t, stream=b)

        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            rec.draw_cull(v, rt)
            a.synchronize()
            if threaded:  # the strictest mode: no thread may make an unsafe call
                g = torch.cuda.CUDAGraph()
                g.capture_begin(capture_error_mode="global")
            else:
                rec.capture_begin()
            rec.draw_cull(v, rt)
            if threaded:
                other = threading.Thread(target=direct)
                other.start()
                other.join()
                g.capture_end()
            else:
                direct()
                g = rec.capture_end()
            rt.commands.zero_()
            g.replay() if threaded else g.launch()
        torch.cuda.synchronize()
        n, recs, _ = O.cull(0, v, small)
        assert_records_equal(rt.read(), (n, recs), "the recorded frame")
        n, cmds, octr, oinst, _ = O.cull_instanced(v, many, ctr, cap, SLOTS)
        assert_records_equal(t.read(), (n, cmds), "the direct call")
        assert np.array_equal(dctr.cpu().numpy().view(np.uint32), octr.view(np.uint32).reshape(-1))
        assert np.array_equal(inst.cpu().numpy().view(np.uint32), oinst)
