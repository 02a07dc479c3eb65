"""The FP64 kernels of grids above the four-lanes-per-face rule (29,184 faces), one face or cell per
thread with loops over the fields, on the states that the small-grid tests use: near vacuum, values of
1e22 and 1e40, NaN, mirror images, NaN-filled scratch, differences and epsilons on both sides of the range
of the float-pair weights.  Exact mode bit for bit against the oracle, fast mode within the one-call
tolerance, as in test_gpu_dropin.py.  The last two tests reach the same arithmetic in the staged and the
fused batch kernels.
"""

import numpy as np
import pytest

from states import noisy, quadrant, smooth
from test_gpu_batch import synced
from test_gpu_dropin import FAST_TOL, STATES, _signed_nan, check, mode, skip_ill_conditioned, tol_for  # noqa: F401
from test_gpu_nan_workspace import _nan_bytes, _nan_out
from test_gpu_solver import oracle_run

pytestmark = pytest.mark.gpu
G = 1.4
LARGE = [(301, 103), (33, 1187)]  # (m-5) n and m (n-5) both above the rule, odd remainders
SMALL = [(8, 8), (13, 22), (31, 17)]  # with a workspace for one sweep they run the same kernels


def ids(s):
    return f"{s[0]}x{s[1]}"


@pytest.mark.parametrize("state", list(STATES))
@pytest.mark.parametrize("shape", LARGE, ids=ids)
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
def test_reconstruction(wx, orc, mode, state, shape, cons):  # noqa: F811
    skip_ill_conditioned(mode, state, cons)
    q = STATES[state](np.random.default_rng(2), *shape)
    for ydir, fw, fo in ((0, wx.weno_x_py, orc.weno_x_py), (1, wx.weno_y_py, orc.weno_y_py)):
        for got, ref, nm in zip(fw(q, G, cons=cons), fo(q, G, cons=cons), ("q_l", "f_l", "q_r", "f_r")):
            check(got, ref, mode, f"{nm} y={ydir}", tol_for(state))


@pytest.mark.parametrize("state", list(STATES))
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
@pytest.mark.parametrize("hlle", [False, True], ids=["blend", "hlle"])
def test_l_local(wx, orc, mode, state, cons, hlle):  # noqa: F811
    skip_ill_conditioned(mode, state, cons, hlle)
    q = STATES[state](np.random.default_rng(5), *LARGE[0])
    args = (0.01, G, hlle, (0.05, 0.4), cons)
    check(wx.l_local_py(q, *args), orc.l_local_py(q, *args), mode, "L", tol_for(state))


def tiny_cells(rng, m, n):
    """Ordinary cells beside cells with subnormal momenta, densities or energies."""
    q = noisy(rng, m, n)
    for k in range(4):
        hit = rng.random((m, n)) < 0.15
        q[hit, k] = rng.choice([-1.0, 1.0], hit.sum()) * 2.0 ** rng.integers(-1074, -1015, hit.sum())
    return q


ENDS = {
    "tiny_cells": tiny_cells,
    "1e-300": lambda rng, m, n: noisy(rng, m, n) * 1e-300,
    "1e-318": lambda rng, m, n: noisy(rng, m, n) * 1e-318,
    "1e-80": lambda rng, m, n: noisy(rng, m, n) * 1e-80,
    "1e76": lambda rng, m, n: noisy(rng, m, n) * 1e76,  # weights d / (eps + beta)^2 near the smallest double
    "1e80": lambda rng, m, n: noisy(rng, m, n) * 1e80,  # subnormal and vanishing weights
    "1e152": lambda rng, m, n: noisy(rng, m, n) * 1e152,
    "1e300": lambda rng, m, n: noisy(rng, m, n) * 1e300,
}


@pytest.mark.parametrize("state", list(ENDS))
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
@pytest.mark.parametrize("shape", [LARGE[0], SMALL[2]], ids=ids)
def test_exact_at_the_ends_of_the_range(wx, orc, state, cons, shape):
    """Quotients with subnormal operands and results, zeros, infinities and NaN inside the loops of the exact
    kernels (and of the four-lane ones): the oracle's bits."""
    q = ENDS[state](np.random.default_rng(77), *shape)
    with np.errstate(all="ignore"):
        for ydir, fw, fo in ((0, wx.weno_x_py, orc.weno_x_py), (1, wx.weno_y_py, orc.weno_y_py)):
            for got, ref, nm in zip(fw(q, G, cons=cons), fo(q, G, cons=cons), ("q_l", "f_l", "q_r", "f_r")):
                check(got, ref, "exact", f"{nm} y={ydir}")
        for hlle in (True, False):
            args = (0.01, G, hlle, (0.05, 0.4), cons)
            check(wx.l_local_py(q, *args), orc.l_local_py(q, *args), "exact", "L")


def _residual(wx, q, cons, hlle, m_, nan_scratch, one_sweep):
    """l_local through the C interface, scratch and output filled with NaN patterns."""
    import torch
    from weno_ext import _lib
    L = _lib.load()
    m, n, c = q.shape
    u = torch.from_numpy(q).cuda()
    wsb = L.weno_l_local_workspace(m, n, int(hlle))
    if one_sweep:
        wsb -= 2 * 4 * 8 * (-(-max((m - 5) * n, m * (n - 5)) // 64) * 64)
    ws = _nan_bytes(torch, wsb) if nan_scratch else torch.zeros(wsb, dtype=torch.uint8, device="cuda")
    out = _nan_out(torch, (m - 6, n - 6, 4))
    _lib.check(L.weno_l_local(u.data_ptr(), m, n, c, *u.stride(), 0.01, G, int(hlle), 0.05, 0.4, int(cons),
                              _lib.FAST if m_ == "fast" else _lib.EXACT, out.data_ptr(), ws.data_ptr(), wsb,
                              torch.cuda.current_stream().cuda_stream), "l_local")
    return out.cpu().numpy()


@pytest.mark.parametrize("state", list(STATES))
@pytest.mark.parametrize("shape", SMALL, ids=ids)
@pytest.mark.parametrize("m_", ["exact", "fast"])
def test_small_grids_through_the_large_grid_kernels(wx, orc, state, shape, m_):
    for cons in (False, True):
        if m_ == "fast" and not cons and state in ("vacuum", "huge", "large"):
            continue  # see skip_ill_conditioned
        q = STATES[state](np.random.default_rng(5), *shape)
        check(_residual(wx, q, cons, True, m_, False, True), orc.l_local_py(q, 0.01, G, True, (0.05, 0.4), cons), m_,
              "L", tol_for(state))


@pytest.mark.parametrize("shape", LARGE, ids=ids)
@pytest.mark.parametrize("cons,hlle", [(False, True), (True, False), (False, False), (True, True)])
def test_l_local_with_nan_scratch(wx, orc, shape, cons, hlle):
    q = noisy(np.random.default_rng(41), *shape)
    ref = orc.l_local_py(q, 0.01, G, hlle, (0.05, 0.4), cons)
    assert np.array_equal(_residual(wx, q, cons, hlle, "exact", True, False), ref)
    check(_residual(wx, q, cons, hlle, "fast", True, False), ref, "fast", "fast")


@pytest.mark.parametrize("ydir", [0, 1], ids=["x", "y"])
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
def test_reconstruct_with_nan_scratch(wx, orc, ydir, cons):
    import torch
    from weno_ext import _lib
    L = _lib.load()
    q = noisy(np.random.default_rng(42), *LARGE[0])
    m, n, c = q.shape
    u = torch.from_numpy(q).cuda()
    ref = (orc.weno_y_py if ydir else orc.weno_x_py)(q, G, cons=cons)
    for m_ in (_lib.EXACT, _lib.FAST):
        outs = [_nan_out(torch, (m - 6, n - 5, 4) if ydir else (m - 5, n - 6, 4)) for _ in range(4)]
        wsb = L.weno_reconstruct_workspace(m, n, ydir)
        ws = _nan_bytes(torch, wsb)
        _lib.check(L.weno_reconstruct(u.data_ptr(), m, n, c, *u.stride(), G, ydir, int(cons), m_,
                                      *[o.data_ptr() for o in outs], ws.data_ptr(), wsb,
                                      torch.cuda.current_stream().cuda_stream), "reconstruct")
        for got, r in zip(outs, ref):
            check(got.cpu().numpy(), r, "exact" if m_ == _lib.EXACT else "fast")


@pytest.mark.parametrize("sign", [1, -1], ids=["+nan", "-nan"])
@pytest.mark.parametrize("cons", [False, True], ids=["char", "cons"])
def test_nan_density_residual(wx, orc, sign, cons):
    q = quadrant(np.random.default_rng(12), 200, 170)
    q[114, 91, 0] = _signed_nan(sign)
    args = (1.0 / 200, G, True, (0.2, 1.0), cons)
    ref = orc.l_local_py(q, *args)
    try:
        check(wx.l_local_py(q, *args), ref, "exact", "exact")
        wx.set_mode("fast")
        fast = wx.l_local_py(q, *args)
    finally:
        wx.set_mode("exact")
    if not cons:
        assert np.isnan(ref[111, 88]).all() and np.isnan(fast[111, 88]).all()
        assert not (np.isnan(ref) & ~np.isnan(fast)).any()
    far = np.ones(ref.shape[:2], dtype=bool)
    far[111 - 4:111 + 5, 88 - 4:88 + 5] = False
    assert np.isfinite(fast[far]).all()
    check(fast[far], ref[far], "fast", "away from the NaN cell")


@pytest.mark.parametrize("ydir", [0, 1], ids=["x", "y"])
def test_fast_reconstruction_mirror_exact(wx, ydir):
    """The wall face between mirror images, component-wise (weno5_cell_fast)."""
    half = noisy(np.random.default_rng(33), 600, 31)
    q = np.concatenate([half[:, ::-1], half], axis=1)
    q[:, :31, 2] *= -1.0
    if ydir == 0:  # the wall across axis 0: exchange the axes and the momenta
        q = np.ascontiguousarray(q.transpose(1, 0, 2)[:, :, [0, 2, 1, 3]])
    wx.set_mode("fast")
    try:
        ql, _, qr, _ = (wx.weno_y_py if ydir else wx.weno_x_py)(np.ascontiguousarray(q), G, cons=True)
    finally:
        wx.set_mode("exact")
    sign = np.array([1.0, 1.0, -1.0, 1.0] if ydir else [1.0, -1.0, 1.0, 1.0])
    wall = (slice(None), 28) if ydir else (28, slice(None))
    assert np.array_equal(ql[wall], qr[wall] * sign)


@pytest.mark.parametrize("log2", [0, 20, 21, 22, 23, 26, 27, 28, 30, 60, -20])
def test_reconstruct_across_the_difference_bound(wx, log2):
    q = noisy(np.random.default_rng(100 + log2), 200, 203)
    q[:, 100:] *= 2.0 ** log2
    for f in (wx.weno_x_py, wx.weno_y_py):
        wx.set_mode("exact")
        ref = f(q, G, cons=True)
        wx.set_mode("fast")
        got = f(q, G, cons=True)
        wx.set_mode("exact")
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= FAST_TOL * np.abs(b).max()


@pytest.mark.parametrize("eps", [1e-20, 2.0 ** -49, 2.0 ** -48, 3.6e-15, 1e-6, 1e3, 2.0 ** 40, 1e14])
@pytest.mark.parametrize("cons", [True, False], ids=["cons", "char"])
def test_step_across_the_epsilon_range(wx, eps, cons):
    q = smooth(np.random.default_rng(7), 186, 196)
    out = []
    for m_ in ("exact", "fast"):
        s = wx.Solver(180, 190, 1 / 190, G, mode=m_, cons=cons, cfl=0.1, weno_eps=eps)
        s.set_state(q[:, :, :4])
        s.run(1)
        out.append(s.state()[..., :4])
    assert np.isfinite(out[0]).all()
    assert np.abs(out[0] - out[1]).max() <= FAST_TOL * np.abs(out[0]).max()


def test_characteristic_blow_up_reproduced(wx, orc):
    """The reference algorithm's own NaN blow-up on a large grid, NaN positions included."""
    q = synced(orc, quadrant(np.random.default_rng(9), 180, 190))
    ref, _, _ = oracle_run(orc, q.copy(), 180, 190, 1 / 190, 0.5, 4, jp=(1e4, 1.1e4), cons=False, hlle=True)
    assert np.isnan(ref).any()
    s = wx.Solver(180, 190, 1 / 190, G, mode="exact", cons=False, force_hlle=True, jp_cri=(1e4, 1.1e4), cfl=0.5)
    s.set_state(q)
    s.run(4)
    got = s.state()
    assert s.info()[2] != 0
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(got[~np.isnan(ref)], ref[~np.isnan(ref)])


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("log2", [0, 21, 22, 23, 24, 40])
def test_batch_across_the_difference_bound(wx, orc, cfg, log2):
    """FP64 tiles and staged kernels, component-wise, one step of quadrant states with 1 % noise in units in
    which the jumps (and from 2^24 on the noise) lie on both sides of 2^22: exact equals the oracle, FAST is
    within the one-call tolerance of it.  (Cell-wise noise is no measure of FAST here: its face states go
    through the density floor and the reference itself reaches 1e113 within the step.)"""
    shapes = [(37, 45), (18, 21)]
    for m_ in ("exact", "fast"):
        b = wx.Batch(20000, 2, precision=64, mode=m_, cons=True, force_hlle=True, cfl=0.2, tile_config=cfg)
        rng = np.random.default_rng(60 + log2)
        for nx, ny in shapes:
            q = quadrant(rng, nx, ny)
            q[..., :4] *= 2.0 ** log2 * (1.0 + 0.01 * rng.random(q.shape[:2])[..., None])
            q = synced(orc, q)
            slot = b.add(q, 1.0 / 45, max_steps=1)
            b.run(1)
            ref = oracle_run(orc, q.copy(), nx, ny, 1.0 / 45, 0.2, 1, cons=True, hlle=True)[0]
            check(b.state(slot)[3:-3, 3:-3, :4], ref[3:-3, 3:-3, :4], m_, m_)
        b.close()


@pytest.mark.parametrize("state", ["noisy", "vacuum", "huge", "large"])
@pytest.mark.parametrize("cfg", [1, 4])
def test_exact_batch_on_extreme_states(wx, orc, state, cfg):
    for cons in (True, False):
        b = wx.Batch(20000, 1, precision=64, mode="exact", cons=cons, force_hlle=False, jp_cri=(0.05, 0.4), cfl=0.2,
                     tile_config=cfg)
        q = synced(orc, STATES[state](np.random.default_rng(8), 37 + 6, 45 + 6))
        slot = b.add(q, 1.0 / 45, max_steps=1)
        b.run(1)
        ref = oracle_run(orc, q.copy(), 37, 45, 1.0 / 45, 0.2, 1, jp=(0.05, 0.4), cons=cons, hlle=False)[0]
        check(b.state(slot)[3:-3, 3:-3, :4], ref[3:-3, 3:-3, :4], "exact", f"{state} cons={cons}")
        b.close()
