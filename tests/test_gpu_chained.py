"""Calls that follow one another on a stream with no synchronisation between, each reading what the
one before it wrote (transforms, depth, pyramid, visibility, counts): launches overlap their
predecessor's end, so a kernel that read too early would show here. Direct calls and a recorded
frame, with and without torch kernels between the calls. Bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, DevicePyramid, Target
from oracle import oracle as O
from tests.helpers import H, W, assert_records_equal, view_for

pytestmark = pytest.mark.gpu

DYN = 1000
STEPS = 6


@pytest.mark.parametrize("form", ["one_call", "kept", "passes"])
@pytest.mark.parametrize("how", ["direct", "torch_between", "recorded"])
def test_frames_chained_without_synchronisation(lib, form, how):
    sc = S.stress_scene(30_011, seed=9, extent=900.0, n_boxes=0)
    boxes = S.make_occluders(np.random.default_rng(4), 60, zmin=150.0, zmax=700.0)
    v = view_for()
    axes = np.tile(np.array([[0.6, 0.0, 0.8]], np.float32), (DYN, 1))
    with Culler(0) as c:
        c.setup_for_rendering(sc)
        dboxes = torch.from_numpy(boxes.reshape(-1)).cuda()
        daxes = torch.from_numpy(axes).cuda()
        ids = torch.arange(DYN, dtype=torch.int32, device="cuda")
        rows = torch.zeros(DYN, 8, dtype=torch.float32, device="cuda")
        depth = torch.zeros(H * W, dtype=torch.float32, device="cuda")
        vis0 = torch.from_numpy(sc.visibility.view(np.int32).copy()).cuda()
        table0 = c.scene_tensors[1].clone()
        vis = vis0.clone()
        pyr = DevicePyramid(W, H)
        t1, t2 = Target.alloc(sc.count), Target.alloc(sc.count)

        def step():
            c.rotate_transforms(ids, daxes, 0.3, rows)
            c.update_object_transform_device(ids, rows)
            if how == "torch_between":
                depth.fill_(1.0)
                vis.add_(0)
            c.raster_boxes(v, dboxes, depth, W, H)
            if form == "one_call":
                c.cull_frame(v, vis, depth, pyr, t1, t2)
            elif form == "kept":
                c.frame_first_pass(v, vis, t1)
                c.generate_depth_pyramid(pyr, depth)
                c.frame_occlusion_pass(pyr, t2)
            else:
                c.draw_cull_first_pass(v, vis, t1)
                c.generate_depth_pyramid(pyr, depth)
                c.draw_cull_occlusion_pass(v, vis, pyr, t2)

        if how == "recorded":
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                step()
                c.capture_begin()
                step()
                g = c.capture_end()
                vis.copy_(vis0)
                c.scene_tensors[1].copy_(table0)
                for _ in range(STEPS):
                    g.launch()
            side.synchronize()
        else:
            for _ in range(STEPS):
                step()
        assert c.check() == 0
        got1, got2 = t1.read(), t2.read()

    ref = S.Scene(sc.objects, sc.transforms.copy(), sc.surfaces, sc.lods)
    opyr = O.pyramid_build(O.depth_raster(v, boxes, W, H))
    ovis = sc.visibility.copy()
    for _ in range(STEPS):
        ref.transforms[:DYN] = O.transforms_rotate(ref.transforms, np.arange(DYN), axes, 0.3)
        n1, r1, _ = O.cull(1, v, ref, vis=ovis)
        n2, r2, _ = O.cull(2, v, ref, vis=ovis, pyramid=opyr)
    assert_records_equal(got1, (n1, r1), f"{form} {how} pass 1")
    assert_records_equal(got2, (n2, r2), f"{form} {how} pass 2")
    assert np.array_equal(vis.cpu().numpy().view(np.uint32), ovis)
    assert np.array_equal(pyr.storage.cpu().numpy().view(np.uint32), opyr.data.view(np.uint32))
