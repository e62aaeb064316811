"""Calls recorded where their stream has just been joined with another, or follows a copy, a fill or nothing: a launch
recorded as a programmatic one then has several nodes before it, or one that is no kernel. Recorded by torch and by the
library, replayed several times; equal to the oracle."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, DevicePyramid, Target
from oracle import oracle as O
from tests.helpers import H, W, assert_records_equal, view_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", ["nothing", "fill", "copy", "host_copy", "join_kernels", "join_copy", "join_library"])
@pytest.mark.parametrize("n", [3000, 60_000])
def test_recorded_after(lib, before, n):
    sc = S.stress_scene(n, seed=9, extent=900.0, n_boxes=0)
    boxes = S.make_occluders(np.random.default_rng(4), 60, zmin=150.0, zmax=700.0)
    v = view_for()
    with Culler(0) as c, Culler(0) as c2:
        c.setup_for_rendering(sc)
        c2.setup_for_rendering(sc)
        source = torch.from_numpy(O.depth_raster(v, boxes, W, H)).cuda()
        host = source.cpu().pin_memory()
        depth, scratch = torch.zeros_like(source), torch.zeros(1 << 22, device="cuda")
        vis0 = torch.from_numpy(sc.visibility.view(np.int32).copy()).cuda()
        vis, vis2 = vis0.clone(), vis0.clone()
        pyr = DevicePyramid(W, H)
        t1, t2, tf, t3 = Target.alloc(n), Target.alloc(n), Target.alloc(n), Target.alloc(n)
        a, b = torch.cuda.Stream(), torch.cuda.Stream()

        def step():
            vis.copy_(vis0)
            if before == "fill":
                scratch.zero_()
                depth.copy_(source)
            elif before == "copy":
                depth.copy_(source)
            elif before == "host_copy":
                depth.copy_(host, non_blocking=True)
            elif before.startswith("join"):
                b.wait_stream(a)
                with torch.cuda.stream(b):
                    scratch.mul_(1.5)
                    if before == "join_copy":
                        depth.copy_(host, non_blocking=True)
                    else:
                        torch.mul(source, 1.0, out=depth)
                    if before == "join_library":
                        c2.draw_cull(v, t3)
                scratch[: 1 << 20].add_(1.0)
                a.wait_stream(b)
            else:
                depth.copy_(source)
            c.draw_cull(v, tf)
            c.draw_cull_first_pass(v, vis, t1)
            c.generate_depth_pyramid(pyr, depth)
            c.draw_cull_occlusion_pass(v, vis, pyr, t2)

        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            step()
            a.synchronize()
            g = torch.cuda.CUDAGraph()
            g.capture_begin(capture_error_mode="thread_local")
            step()
            g.capture_end()
            for t in (t1, t2, tf, t3):
                t.commands.zero_()
            depth.zero_()
            for _ in range(3):
                g.replay()
            torch.cuda.synchronize()
            assert c.check() == 0
            ovis, opyr = sc.visibility.copy(), O.pyramid_build(source.cpu().numpy())
            nf, rf, _ = O.cull(0, v, sc)
            n1, r1, _ = O.cull(1, v, sc, vis=ovis)
            n2, r2, _ = O.cull(2, v, sc, vis=ovis, pyramid=opyr)
            assert_records_equal(tf.read(), (nf, rf), "frustum")
            assert_records_equal(t1.read(), (n1, r1), "pass 1")
            assert_records_equal(t2.read(), (n2, r2), "pass 2")
            if before == "join_library":
                assert_records_equal(t3.read(), (nf, rf), "the other stream's")
            assert np.array_equal(vis.cpu().numpy().view(np.uint32), ovis)
