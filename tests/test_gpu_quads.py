"""Face kernels on both sides of the four-lanes-per-face rule (29,184 faces): the residual and the
reconstruction of grids just below and just above it against the oracle, bit for bit in exact mode
and within the one-call tolerance (1e-11 of the largest magnitude) in fast mode, ragged extents and
the smallest grid included."""

import numpy as np
import pytest

from states import noisy, quadrant

pytestmark = pytest.mark.gpu
G = 1.4
TOL = 1e-11


@pytest.fixture(scope="module")
def wx():
    import weno_ext
    yield weno_ext
    weno_ext.set_mode("exact")


# (m, n) of the array; x faces (m-5) n and y faces m (n-5) straddle the rule one by one
SHAPES = [(8, 8), (9, 41), (171, 176), (176, 171), (177, 172), (301, 97), (33, 1021), (200, 203)]


@pytest.mark.parametrize("mn", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("cons", [True, False], ids=["cons", "char"])
@pytest.mark.parametrize("hlle", [True, False], ids=["hlle", "blend"])
def test_residual(wx, orc, mn, cons, hlle):
    rng = np.random.default_rng(sum(mn))
    q = quadrant(rng, mn[0] - 6, mn[1] - 6)
    q[..., :4] *= 1.0 + 0.01 * rng.random(q.shape[:2])[..., None]
    args = (0.01, G, hlle, (0.2, 1.0), cons)
    ref = orc.l_local_py(q, *args)
    wx.set_mode("exact")
    assert np.array_equal(wx.l_local_py(q, *args), ref)
    wx.set_mode("fast")
    assert np.abs(wx.l_local_py(q, *args) - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("mn", SHAPES[1:4], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("ydir", [False, True], ids=["x", "y"])
def test_reconstruct(wx, orc, mn, ydir):
    q = noisy(np.random.default_rng(mn[0]), *mn)
    for cons in (True, False):
        ref = (orc.weno_y_py if ydir else orc.weno_x_py)(q, G, cons=cons)
        wx.set_mode("exact")
        got = (wx.weno_y_py if ydir else wx.weno_x_py)(q, G, cons=cons)
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
