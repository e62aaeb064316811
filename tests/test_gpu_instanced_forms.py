"""The instanced cull over LOD counts at the edges of its block sizes (a row of counts per warp: 32, 16 or 8
warps a block; more or fewer LODs than threads), over list sizes from nothing to several groups, and in
the form a recorded call of many LODs takes. Counters, instance lists and commands equal the oracle's."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.abi import BlzError
from blitzen_gb300.culler import Culler, Target
from oracle import oracle as O
from tests.helpers import assert_records_equal, view_for

pytestmark = pytest.mark.gpu

SLOTS = 700


def _scene(n, lods, seed=4, extent=900.0):
    """n objects over `lods` single-LOD surfaces (a surface of the last one has what is left)."""
    rng = np.random.default_rng(seed)
    meshes = max(1, lods // 3)
    objs, tr = S.make_objects(rng, n, extent, meshes)
    surf = np.zeros(meshes, abi.PRIMITIVE_SURFACE)
    surf["center"] = rng.uniform(-1, 1, (meshes, 3))
    surf["radius"] = rng.uniform(0.5, 3.0, meshes)
    surf["lodOffset"] = np.arange(meshes) * (lods // meshes)
    surf["lodCount"] = lods // meshes
    table = np.zeros(lods, abi.LOD_DATA)
    table["indexCount"] = np.arange(lods) + 3
    table["firstIndex"] = np.arange(lods) * 7
    table["error"] = rng.choice(np.array([0.0, 0.02, 0.1, 0.5], np.float32), lods)
    return S.Scene(objs, tr, surf, table)


def _check(c, sc, v, run=None, slots=SLOTS):
    cap = len(sc.lods) * slots
    ctr = O.new_counters(sc, slots)
    dctr = torch.from_numpy(ctr.view(np.int32).reshape(-1).copy()).cuda()
    inst = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    t = Target.alloc(len(sc.lods))
    call = lambda: c.draw_instance_cull_pass(v, dctr, inst, slots, t)  # noqa: E731
    (run or (lambda f: f()))(call)
    flags = c.flags()
    n, cmds, octr, oinst, oflags = O.cull_instanced(v, sc, ctr, cap, slots)
    assert flags == oflags
    assert_records_equal(t.read(), (n, cmds), "commands")
    assert np.array_equal(dctr.cpu().numpy().view(np.uint32), octr.view(np.uint32).reshape(-1))
    assert np.array_equal(inst.cpu().numpy().view(np.uint32), oinst)


@pytest.mark.parametrize("lods", [1, 3, 33, 256, 511, 1023, 1024, 1025, 1462, 1463, 2000, 2694, 2695, 4095, 4096])
def test_lod_counts(lib, lods):
    with Culler(0) as c:
        sc = _scene(30_001, lods)
        c.setup_for_rendering(sc)
        for pos in ((0.0, 0.0, 0.0), (100.0, 20.0, -700.0)):
            _check(c, sc, view_for(position=pos))


@pytest.mark.parametrize("lods", [48, 1200])
@pytest.mark.parametrize("n", [1, 31, 64, 65, 2047, 2049, 70_000, 400_003])
def test_list_sizes(lib, n, lods):
    with Culler(0) as c:
        sc = _scene(n, lods, extent=60.0 if n < 100 else 900.0)
        c.setup_for_rendering(sc)
        for slots in (SLOTS, 3):  # lists that overflow too
            _check(c, sc, view_for(), slots=slots)


@pytest.mark.parametrize("warm", [False, True])
def test_many_lods_recorded(lib, warm):
    with Culler(0) as c:
        sc = _scene(30_001, 1500)
        c.setup_for_rendering(sc)
        side = torch.cuda.Stream()

        def recorded(call):
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                if warm:
                    call()
                c.capture_begin()
                call()
                g = c.capture_end()
                g.launch()
                g.launch()
            side.synchronize()

        _check(c, sc, view_for(), recorded)
        big = _scene(200_000, 1500)  # and the direct form after it, with more scratch
        c.setup_for_rendering(big)
        _check(c, big, view_for())


def test_too_many_lods_refused(lib):
    with Culler(0) as c:
        sc = _scene(1000, 4097)
        c.setup_for_rendering(sc)
        with pytest.raises(BlzError):
            _check(c, sc, view_for())
