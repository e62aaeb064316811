"""The pyramid's tile build at the extents where its parts meet (tile remainders, one-wide levels, odd
levels, the three widths of depth load, paired and single texel stores), alone and inside the one-call
frame. Every texel equals the oracle's bit for bit, NaN, -0.0 and negative depths among the inputs."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import abi
from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler, DevicePyramid, Target
from oracle import oracle as O
from tests.helpers import view_for

pytestmark = pytest.mark.gpu

EXTENTS = [(1, 1), (2, 2), (3, 2), (5, 3), (4, 130), (64, 64), (66, 62), (65, 129), (128, 2), (130, 258), (257, 255), (1366, 768),
           (1919, 1079), (4100, 6), (6, 4100), (2560, 1440), (3840, 2160)]
ALIGN = {"16": 0, "8": 2, "4": 1}  # floats the depth buffer starts past a 16-byte boundary


def _depth(w, h, odd):
    rng = np.random.default_rng(w * 7919 + h)
    d = rng.random((h, w)).astype(np.float32)
    if odd:
        flat = d.reshape(-1)
        k = rng.integers(0, w * h, max(1, w * h // 9))
        flat[k] = rng.choice(np.array([np.nan, -0.0, 0.0, -1.0, np.inf, -np.inf], np.float32), len(k))
    return d


def _device(d, shift):
    t = torch.zeros(d.size + 4, dtype=torch.float32, device="cuda")[shift:shift + d.size]
    t.copy_(torch.from_numpy(d.reshape(-1)))
    return t


@pytest.fixture(scope="module")
def c(lib):
    with Culler(0) as c:
        yield c


@pytest.mark.parametrize("mode", [abi.HIZ_D3D12, abi.HIZ_VULKAN])
@pytest.mark.parametrize("align", list(ALIGN))
@pytest.mark.parametrize("extent", EXTENTS, ids=lambda e: f"{e[0]}x{e[1]}")
def test_every_texel(c, extent, align, mode):
    w, h = extent
    for odd in (False, True):
        d = _depth(w, h, odd)
        pyr = DevicePyramid(w, h, mode)
        pyr.storage.fill_(7.0)
        if align == "4":  # texel storage off the 8-byte boundary too
            keep = torch.full((pyr.storage.numel() + 1,), 7.0, dtype=torch.float32, device="cuda")
            pyr.storage = keep[1:]
            pyr.desc.data = pyr.storage.data_ptr()
        c.generate_depth_pyramid(pyr, _device(d, ALIGN[align]))
        ref = O.pyramid_build(d, mode).data
        got = pyr.storage.cpu().numpy()
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), (extent, mode, odd, np.nonzero(got.view(np.uint32) != ref.view(np.uint32))[0][:4])


@pytest.mark.parametrize("mode", [abi.HIZ_D3D12, abi.HIZ_VULKAN])
@pytest.mark.parametrize("extent", [(66, 62), (1366, 768), (1919, 1079)], ids=lambda e: f"{e[0]}x{e[1]}")
@pytest.mark.parametrize("threads,opt", [(256, 2), (128, 2), (512, 1)])
def test_inside_the_frame_kernel(lib, extent, mode, threads, opt):
    w, h = extent
    sc = S.stress_scene(3001, seed=2, extent=300.0, n_boxes=0)
    d = _depth(w, h, False)
    with Culler(0) as c:
        c.set_launch_shape(threads, opt)
        c.setup_for_rendering(sc)
        pyr = DevicePyramid(w, h, mode)
        v = view_for(width=w, height=h, pw=float(pyr.desc.width), ph=float(pyr.desc.height))
        vis = torch.from_numpy(sc.visibility.view(np.int32).copy()).cuda()
        t1, t2 = Target.alloc(sc.count), Target.alloc(sc.count)
        c.cull_frame(v, vis, _device(d, 0), pyr, t1, t2)
        assert c.check() == 0
    opyr = O.pyramid_build(d, mode)
    ovis = sc.visibility.copy()
    n1, _, _ = O.cull(1, v, sc, vis=ovis)
    n2, _, _ = O.cull(2, v, sc, vis=ovis, pyramid=opyr)
    assert np.array_equal(pyr.storage.cpu().numpy().view(np.uint32), opyr.data.view(np.uint32))
    assert (t1.read()[0], t2.read()[0]) == (n1, n2)
    assert np.array_equal(vis.cpu().numpy().view(np.uint32), ovis)


def test_vulkan_descriptor_of_any_extent(c):
    """A caller's own descriptor whose mip 0 is not a power of two: every level after the sampler's rule."""
    d = _depth(150, 91, False)
    pyr, host = DevicePyramid(300, 182, abi.HIZ_D3D12), O.HostPyramid(300, 182, abi.HIZ_D3D12)  # 150 x 91 levels
    for desc in (pyr.desc, host.desc):
        desc.mode, desc.depthWidth, desc.depthHeight = abi.HIZ_VULKAN, 150, 91
    c.generate_depth_pyramid(pyr, _device(d, 0))
    ref = O.pyramid_build(d, abi.HIZ_VULKAN, into=host)
    assert np.array_equal(pyr.storage.cpu().numpy().view(np.uint32), ref.data.view(np.uint32))
