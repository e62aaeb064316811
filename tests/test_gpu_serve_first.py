"""The first requests of a process's first server wait for no kernel to be loaded. In a process of its own, since a
loaded kernel stays loaded."""
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C, time, numpy as np, torch
from blitzen_gb300 import abi, scenes as S
from blitzen_gb300.culler import Culler
from tests.helpers import view_for
with Culler(0) as c:
    c.setup_for_rendering(S.frustum_lod_scene(50_000))
    cfg, server = abi.ServeConfig(1 << 30, 4, 64, 1000, abi.STRIDE_VULKAN), C.c_void_p()
    abi.check(c.lib.blz_serve_create(c.ctx, C.byref(cfg), C.byref(server)), "create")
    axes = np.tile(np.array([[0.0, 0.6, 0.8]], np.float32), (1000, 1))
    worst = 0.0
    for k in range(8):
        r, t, res = abi.ServeRequest(), C.c_uint64(), abi.ServeResult()
        r.view, r.mode, r.list = view_for(yaw=0.1 * k), 0, abi.RenderList(c.scene_tensors[0].data_ptr(), 30_000)
        r.rotateCount, r.rotateAxes, r.rotateAngle, r.copyToHost = 1000, axes.ctypes.data, 0.01, 0
        t0 = time.perf_counter()
        abi.check(c.lib.blz_serve_submit(server, C.byref(r), C.byref(t)), "submit")
        abi.check(c.lib.blz_serve_wait(server, t, 10_000, C.byref(res)), "wait")
        worst = max(worst, time.perf_counter() - t0)
        assert res.status == 0
        c.lib.blz_serve_release(server, t)
    c.lib.blz_serve_destroy(server)
    print("worst_ms", worst * 1e3)
"""


def test_first_requests_load_no_kernel(lib):
    out = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    ms = float(out.stdout.split("worst_ms")[1])
    assert ms < 6.0, ms  # 21 with every kernel loaded by its first launch, 13 when a batch had two kernels
