"""The tile raster with boxes sorted into bins (many boxes over many tiles): on both sides of the rule, images that
are no multiple of a tile or of the bins, one bin wide or high, a bin holding more boxes than a tile's list, and
boxes of every size. Bit-exact against the oracle; and many tiny boxes over a large image take no longer than a
launch per box did."""
import numpy as np
import pytest
import torch

from blitzen_gb300 import scenes as S
from blitzen_gb300.culler import Culler
from oracle import oracle as O
from tests.helpers import view_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def c(lib):
    with Culler(0) as c:
        yield c


def _check(c, boxes, w, h):
    v = view_for(width=w, height=h)
    room = torch.full((w * h + 64,), 5.0, dtype=torch.float32, device="cuda")
    c.raster_boxes(v, torch.from_numpy(boxes.reshape(-1)).cuda(), room[:w * h], w, h)
    got = room.cpu().numpy()
    assert np.array_equal(got[:w * h].view(np.uint32), O.depth_raster(v, boxes, w, h).reshape(-1).view(np.uint32))
    assert (got[w * h:] == 5.0).all()


@pytest.mark.parametrize("count,w,h", [(1536, 4097, 3300), (1537, 4097, 3300), (2298, 4096, 2176), (2297, 4096, 2176), (3000, 4001, 2301),
                                       (8192, 2600, 1000), (8191, 65536, 60), (8192, 50, 65500), (8192, 3841, 2161)])
def test_rule_and_extents(c, count, w, h):
    _check(c, S.make_occluders(np.random.default_rng(count), count, size=(1.0, 60.0)), w, h)


@pytest.mark.parametrize("size", [(0.5, 2.0), (500.0, 3000.0)])
def test_sizes(c, size):
    _check(c, S.make_occluders(np.random.default_rng(7), 4000, size=size), 4000, 2200)


def test_more_boxes_in_a_bin_than_a_list_holds(c):
    rng = np.random.default_rng(1)
    b = S.make_occluders(rng, 5000, zmin=20.0, zmax=400.0, size=(0.05, 1.0), half_fov_tan=(0.04, 0.04))
    far = S.make_occluders(rng, 1000)
    _check(c, np.concatenate([b, far])[rng.permutation(6000)], 4000, 2200)


def test_time_of_tiny_boxes_over_a_large_image(c):
    """8,192 boxes of 1 to 4 units at 8192x8192: clearing the image and a block per box took 74 us, every tile testing
    every box 140."""
    w = h = 8192
    v, d = view_for(width=w, height=h), torch.zeros(h, w, device="cuda")
    b = torch.from_numpy(S.make_occluders(np.random.default_rng(2), 8192, size=(1.0, 4.0)).reshape(-1)).cuda()
    best = 1e9
    for _ in range(10):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        for _ in range(10):
            c.raster_boxes(v, b, d, w, h)
        e.record()
        torch.cuda.synchronize()
        best = min(best, s.elapsed_time(e) * 100.0)
    assert best < 100.0, best
