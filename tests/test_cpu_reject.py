"""The bound behind the kernels' reject test, restated in numpy: over rough transforms (NaN, infinities,
quaternions of any length, negative scales, spheres within rounding of the planes) no object it drops is
one the oracle's exact frustum test keeps, and over an ordinary scene it drops nearly all that are outside."""
import numpy as np
import pytest

from blitzen_gb300 import scenes as S
from oracle import oracle as O
from tests.helpers import view_for
from tests.test_gpu_reject import VIEWS, rough_scene

F = np.float32
ULPS = F(2.0 ** -18)


def _fma(a, b, c):  # one rounding (a float64 product of floats is exact; its sum is off by less than the bound allows)
    return (a.astype(np.float64) * np.float64(b) + np.asarray(c, np.float64)).astype(F)


def dropped(v, sc) -> np.ndarray:
    n, rows = sc.count, sc.transforms.view(F).reshape(-1, 8)
    tid, sid = sc.objects["transformId"].astype(np.int64), sc.objects["surfaceId"].astype(np.int64)
    known = (tid < len(rows)) & (sid < len(sc.surfaces))
    t, s = rows[np.where(known, tid, 0)], sc.surfaces[np.where(known, sid, 0)]
    off, cnt = s["lodOffset"].astype(np.int64), s["lodCount"].astype(np.int64)
    known &= (off < len(sc.lods)) & (cnt <= len(sc.lods) - off)
    m = np.array(v.viewMatrix, F).reshape(4, 4)  # column-major: row k is m[:, k]
    r = [m[:, k] for k in range(3)]
    norm = [F(np.sqrt(np.sum(x[:3].astype(np.float64) ** 2))) for x in r]
    fl, fr, fb, ft = (abs(F(x)) for x in (v.frustumLeft, v.frustumRight, v.frustumBottom, v.frustumTop))
    span = max(F(1), fl + fr, fb + ft)
    big, far = max(np.abs(x[:3]).max() for x in r), max(abs(x[3]) for x in r)
    a = F(1.001953125) * max(norm[2], fl * norm[2] + fr * norm[0], fb * norm[2] + ft * norm[1]) + F(1e-18)
    b, d = ULPS * span * big, ULPS * span * far + F(1e-30)
    with np.errstate(all="ignore"):
        x, y, z = (_fma(t[:, 0], k[0], _fma(t[:, 1], k[1], _fma(t[:, 2], k[2], k[3]))) for k in r)
        q = t[:, 4:]
        nn = ((q[:, 3] * q[:, 3]).astype(F) + q[:, 2] ** 2 + q[:, 1] ** 2 + q[:, 0] ** 2).astype(F)
        k = np.fmax(F(1), F(2) * nn - F(1))
        rad = s["radius"] * t[:, 3]
        c = np.abs(s["center"]).sum(axis=1, dtype=F)
        top = rad + ULPS * np.abs(rad) + d + b * (np.abs(t[:, 0]) + np.abs(t[:, 1]) + np.abs(t[:, 2])) + a * (np.abs(t[:, 3]) * c * k)
        side = z * F(v.frustumLeft) - np.abs(x) * F(v.frustumRight)
        updown = z * F(v.frustumBottom) - np.abs(y) * F(v.frustumTop)
        low = np.fmin(np.fmin(side, updown), np.fmin(z - F(v.zNear), F(v.zFar) - z))
        return known & (low < -top)


@pytest.mark.parametrize("k", range(len(VIEWS)))
@pytest.mark.parametrize("seed", [1, 2])
def test_never_drops_a_visible_object(k, seed):
    sc = rough_scene(60, n=20_000, seed=seed)
    v = view_for(**VIEWS[k])
    _, recs, _ = O.cull(0, v, sc)
    out = dropped(v, sc)
    assert not out[recs[:, 0].astype(np.int64)].any()
    assert out.any()


def test_drops_nearly_all_that_are_outside():
    sc = S.frustum_lod_scene(50_000, seed=0)
    v = view_for()
    n, recs, _ = O.cull(0, v, sc)
    assert dropped(v, sc).sum() > 0.99 * (sc.count - n)
