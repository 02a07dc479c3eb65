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


@pytest.mark.parametrize("mn", [(8, 8), (9, 41), (150, 160)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("hlle", [True, False], ids=["hlle", "blend"])
def test_workspace_for_one_sweep(wx, mn, hlle):
    """A workspace without the second sweep's pass-1 planes runs the sweeps in turn, to the same
    bits; a smaller one is refused."""
    import torch
    from weno_ext import _lib
    L = _lib.load()
    m, n = mn
    q = torch.from_numpy(quadrant(np.random.default_rng(m), m - 6, n - 6)).cuda()
    full = L.weno_l_local_workspace(m, n, int(hlle))
    p1 = -(-max((m - 5) * n, m * (n - 5)) // 64) * 64  # planes are padded to 64 values
    one = full - 2 * 4 * 8 * p1
    outs = []
    for wsb in (full, one, one - 256):
        out = torch.zeros((m - 6, n - 6, 4), dtype=torch.float64, device="cuda")
        ws = torch.zeros(full, dtype=torch.uint8, device="cuda")
        rc = L.weno_l_local(q.data_ptr(), m, n, q.shape[2], *q.stride(), 0.01, G, int(hlle), 0.2, 1.0, 0, _lib.EXACT,
                            out.data_ptr(), ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream)
        outs.append((rc, out.cpu().numpy()))
    assert outs[0][0] == 0 and outs[1][0] == 0 and outs[2][0] != 0
    assert np.abs(outs[0][1]).max() > 0
    assert np.array_equal(outs[0][1], outs[1][1])
