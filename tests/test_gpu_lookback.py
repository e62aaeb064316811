"""The bounded look-back of the instanced cull of many LODs, in the recorded form that waits: its waits run
out when its ticket has been advanced, and the replay after that equals the oracle. A direct call after the
hook takes that form as well (one launch), the one after it the counting sort again (four); so does a call of a
few objects, which are one tile and wait for none."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, Target, to_device
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu

SLOTS = 5_000


class Pass:
    def __init__(self, c):
        self.sc, self.v, self.c = S.frustum_lod_scene(60_000, seed=5, n_meshes=300, extent=800.0), view_for(zfar=1e4), c
        assert len(self.sc.lods) > 1024
        c.setup_for_rendering(self.sc)
        self.ctr = O.new_counters(self.sc, SLOTS)
        self.cap = len(self.sc.lods) * SLOTS
        self.dctr = torch.from_numpy(self.ctr.view(np.int32).reshape(-1).copy()).cuda()
        self.inst = torch.full((self.cap,), -1, dtype=torch.int32, device="cuda")
        self.t = Target.alloc(len(self.sc.lods))

    def call(self):
        self.c.draw_instance_cull_pass(self.v, self.dctr, self.inst, SLOTS, self.t)

    def clear(self):
        self.inst.fill_(-1)
        self.t.commands.zero_()

    def check(self):
        n, cmds, octr, oinst, _ = O.cull_instanced(self.v, self.sc, self.ctr, self.cap, SLOTS)
        assert_records_equal(self.t.read(), (n, cmds), "commands")
        assert np.array_equal(self.dctr.cpu().numpy().view(np.uint32), octr.view(np.uint32).reshape(-1))
        assert np.array_equal(self.inst.cpu().numpy().view(np.uint32), oinst)


@pytest.mark.parametrize("advance", [1, 4])
def test_recorded_lookback_runs_out_then_recovers(lib, advance):
    with Culler(0) as c:
        p = Pass(c)
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            graphs = []
            for polls in (16, 0):  # the limit is part of the recorded launch; 0: the default
                c.set_wait_limit(polls)
                c.capture_begin()
                p.call()
                graphs.append(c.capture_end())
            c.debug_advance_ticket(advance)
            graphs[0].launch()
            assert c.flags() & abi.FLAG_TIMEOUT
            p.clear()
            graphs[1].launch()
            assert c.check() == 0
        p.check()


@pytest.mark.parametrize("n,launches", [(1, 1), (32, 1), (128, 1), (129, 4), (5000, 4)])
def test_few_objects_take_one_launch(lib, n, launches):
    with Culler(0) as c:
        p = Pass(c)
        objs = np.ascontiguousarray(p.sc.objects[:n])
        d = to_device(objs, "cuda")
        before = c.launches
        c.draw_instance_cull_pass(p.v, p.dctr, p.inst, SLOTS, p.t, objects=d, count=n)
        assert c.launches - before == launches
        assert c.check() == 0
        cnt, cmds, octr, oinst, _ = O.cull_instanced(p.v, p.sc, p.ctr, p.cap, SLOTS, objects=objs)
        assert_records_equal(p.t.read(), (cnt, cmds), "commands")
        assert np.array_equal(p.dctr.cpu().numpy().view(np.uint32), octr.view(np.uint32).reshape(-1))
        assert np.array_equal(p.inst.cpu().numpy().view(np.uint32), oinst)


def test_direct_call_after_the_hook_takes_the_waiting_form(lib):
    with Culler(0) as c:
        p = Pass(c)
        launches = []
        for hook in (False, True, False):
            c.set_wait_limit(16 if hook else 0)
            if hook:
                c.debug_advance_ticket(2)
            p.clear()
            before = c.launches
            p.call()
            launches.append(c.launches - before)
            assert (c.flags() & abi.FLAG_TIMEOUT != 0) == hook
        assert launches == [4, 1, 4]
        p.check()
