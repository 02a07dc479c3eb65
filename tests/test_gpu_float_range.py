"""The reciprocal WENO weights of the FP32 and df64 kernels at the ends of the float exponent range: 1 / (eps +
beta)^2 of a vanishing epsilon (a locally uniform flow whose shear field takes eps rho^2, or a small weno_eps)
and of large differences.

Tolerances against the native FP64 exact solver after two steps, relative L1 per conserved channel: 1e-10 for
df64 and 1e-5 for FP32, as everywhere else.
"""

import numpy as np
import pytest

from states import rel_l1

pytestmark = pytest.mark.gpu
G = 1.4
TOL = {"df64": 1e-10, 32: 1e-5}


def flow(scale, n=40, amp=0.1):
    """Smooth waves on one half of the domain, uniform on the other; density, momentum and energy of order
    `scale` (velocities and sound speeds of order one)."""
    x = (np.arange(n + 6) + 0.5) / (n + 6)
    w = np.where(x < 0.5, 0.0, np.sin(4 * np.pi * (x - 0.5)) ** 2)
    w = amp * w[:, None] * w[None, :]
    rho, u, v, p = 1 + w, 0.4 + w, -0.3 - 0.5 * w, 1 + 0.5 * w
    q = np.stack([rho, rho * u, rho * v, p / (G - 1) + 0.5 * rho * (u * u + v * v)], axis=-1)
    return np.ascontiguousarray(q * scale)


def run(wx, q, precision, eps, cons, mode="fast"):
    n = q.shape[0] - 6
    s = wx.Solver(n, n, 1 / n, G, precision=precision, mode=mode, cons=cons, cfl=0.4, weno_eps=eps)
    s.set_state(q)
    s.run(2)
    return s.state()[3:-3, 3:-3, :4]


@pytest.mark.parametrize("precision", ["df64", 32])
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
@pytest.mark.parametrize("scale,eps", [(2e-6, 1e-12), (1e-9, 1e-12), (1.0, 1e-24), (1.0, 1e-36), (1e-5, 1e-30)],
                         ids=lambda x: f"{x:g}")
def test_vanishing_epsilon(wx, precision, cons, scale, eps):
    q = flow(scale)
    ref = run(wx, q, 64, eps, cons, "exact")
    got = run(wx, q, precision, eps, cons)
    assert np.isfinite(got).all()
    for c in range(4):
        assert rel_l1(got[..., c], ref[..., c]) <= TOL[precision], c


@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
@pytest.mark.parametrize("scale", [1e8, 1e12])
def test_large_differences_df64(wx, cons, scale):
    """Differences whose fourth power passes the largest float (2^128)."""
    q = flow(scale)
    ref = run(wx, q, 64, 1e-12, cons, "exact")
    got = run(wx, q, "df64", 1e-12, cons)
    assert np.isfinite(got).all()
    for c in range(4):
        assert rel_l1(got[..., c], ref[..., c]) <= TOL["df64"], c


@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
def test_fp32_below_its_range_takes_linear_weights(wx, cons):
    """Indicators whose squares vanish in FP32 (states of order 1e-9 with an epsilon to match): the weights
    are the linear ones, those of native FP64 with an epsilon far above every indicator."""
    q = flow(1e-9)
    ref = run(wx, q, 64, 1.0, cons, "exact")
    got = run(wx, q, 32, 1e-30, cons)
    for c in range(4):
        assert rel_l1(got[..., c], ref[..., c]) <= TOL[32], c
