"""FAST FP64 reconstruction where the float-pair weights (csrc/ffw.cuh) hand over to the FP64 ones:
differences on both sides of 2^22 in one array, and epsilons on both sides of the covered range.
FAST against exact within the one-call tolerance (1e-11 of the largest magnitude)."""

import numpy as np
import pytest

from states import noisy, smooth

pytestmark = pytest.mark.gpu
G = 1.4
TOL = 1e-11


@pytest.fixture(scope="module")
def wx():
    import weno_ext
    yield weno_ext
    weno_ext.set_mode("exact")


@pytest.mark.parametrize("log2", [0, 20, 21, 22, 23, 26, 27, 28, 30, -20])
def test_reconstruct_across_the_difference_bound(wx, log2):
    # component-wise: across a jump of 2^20 the characteristic matrices and the limiter
    # turn one rounding of the input into per cents of the state
    rng = np.random.default_rng(100 + log2)
    q = noisy(rng, 37, 41)
    q[:, 20:] *= 2.0 ** log2  # both ranges, and faces whose stencils hold both
    for f in (wx.weno_x_py, wx.weno_y_py):
        wx.set_mode("exact")
        ref = f(q, G, cons=True)
        wx.set_mode("fast")
        got = f(q, G, cons=True)
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("eps", [1e-20, 2.0 ** -58, 3e-18, 1e-6, 1e3, 2.0 ** 40, 1e14])
@pytest.mark.parametrize("cons", [True, False], ids=["cons", "char"])
def test_step_across_the_epsilon_range(wx, eps, cons):
    rng = np.random.default_rng(7)
    q = smooth(rng, 30, 34)
    out = []
    for mode in ("exact", "fast"):
        s = wx.Solver(24, 28, 1 / 28, G, mode=mode, cons=cons, cfl=0.1, weno_eps=eps)
        s.set_state(q[:, :, :4])
        s.run(1)
        out.append(s.state()[..., :4])
    assert np.isfinite(out[0]).all()
    assert np.abs(out[0] - out[1]).max() <= TOL * np.abs(out[0]).max()
