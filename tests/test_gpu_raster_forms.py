"""The box raster by screen tiles and by boxes, at the sizes where each can go wrong: extents that are no
multiple of the tile or of four, buffers off the 16-byte boundary, no box, more boxes over one tile than
its list holds, and more boxes than the tile form takes. Bit-exact against the oracle, and nothing
outside the image is written."""
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


def _check(c, boxes, w, h, shift=0):
    v = view_for(width=w, height=h)
    room = torch.full((w * h + 64,), 5.0, dtype=torch.float32, device="cuda")
    depth = room[shift:shift + w * h]
    c.raster_boxes(v, torch.from_numpy(boxes.reshape(-1)).cuda(), depth, w, h)
    got = room.cpu().numpy()
    ref = O.depth_raster(v, boxes, w, h)
    assert np.array_equal(got[shift:shift + w * h].view(np.uint32), ref.reshape(-1).view(np.uint32))
    assert (got[:shift] == 5.0).all() and (got[shift + w * h:] == 5.0).all()


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("extent", [(1, 1), (63, 65), (64, 64), (68, 130), (257, 7), (1366, 768), (1919, 1079)], ids=lambda e: f"{e[0]}x{e[1]}")
def test_extents(c, extent, shift):
    _check(c, S.make_occluders(np.random.default_rng(3), 300, zmin=50.0, zmax=900.0), *extent, shift)


@pytest.mark.parametrize("count", [0, 1, 255, 257, 1025, 4096, 8192, 8193])
def test_counts(c, count):
    _check(c, S.make_occluders(np.random.default_rng(count), count), 640, 360)


@pytest.mark.parametrize("count", [513, 3000])
def test_all_boxes_over_one_tile(c, count):
    rng = np.random.default_rng(1)
    b = S.make_occluders(rng, count, zmin=20.0, zmax=400.0, size=(1.0, 30.0), half_fov_tan=(0.05, 0.05))
    _check(c, b, 512, 512)


def test_boxes_behind_and_across_the_near_plane(c):
    b = S.make_occluders(np.random.default_rng(2), 400, zmin=-300.0, zmax=300.0)
    _check(c, b, 320, 200)
