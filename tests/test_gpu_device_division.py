"""The integer FP64 quotient and square root (csrc/rn64.cuh) on the device, with the hardware seeds: bit for bit
the IEEE results.  1/x and sqrt(x) through weno_fast_math_eval over all exponents, subnormals, specials and
all-ones significands; a/b through the exact con2primi (u = q1 / rho for rho above the 1e-12 floor), with
near-half-way quotients and results at both ends of the range."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _doubles(rng, n, lo=0, hi=2047):
    bits = rng.integers(0, 2 ** 52, n, dtype=np.uint64) | (rng.integers(lo, hi, n, dtype=np.uint64) << np.uint64(52))
    ones = rng.random(n) < 0.1
    bits[ones] |= np.uint64(2 ** 52 - 1)
    return bits.view(np.float64)


def test_reciprocal_and_root_bit_for_bit(wx):
    import torch
    from weno_ext import _lib
    L = _lib.load()
    rng = np.random.default_rng(5)
    x = np.concatenate([_doubles(rng, 400000), _doubles(rng, 50000, 0, 1), _doubles(rng, 50000, 1018, 1029),
                        np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** -1074 * 3,
                                  np.finfo(float).max, 1.0, 4.0, 2.0 ** -1023])])
    x = np.concatenate([x, -x[:100000]])
    xd = torch.from_numpy(x).cuda()
    out = torch.empty(4 * x.size, dtype=torch.float64, device="cuda")
    _lib.check(L.weno_fast_math_eval(xd.data_ptr(), out.data_ptr(), x.size,
                                     torch.cuda.current_stream().cuda_stream), "eval")
    o = out.cpu().numpy().reshape(4, -1)
    with np.errstate(all="ignore"):
        for got, want in ((o[0], 1.0 / x), (o[2], np.sqrt(x))):
            assert np.array_equal(np.isnan(got), np.isnan(want))
            fin = ~np.isnan(want)
            assert np.array_equal(got[fin].view(np.uint64), want[fin].view(np.uint64))


def test_quotient_bit_for_bit(wx):
    rng = np.random.default_rng(6)
    m, n = 400, 500
    rho = _doubles(rng, m * n, 1023 - 39, 2046)
    num = _doubles(rng, m * n)
    half = rng.random(m * n) < 0.3  # within rounding of rho times a short number: near half-way quotients
    num[half] = (_doubles(rng, m * n, 1023 - 2, 1023 + 2) * (rho * 2.0 ** -40))[half]
    num[rng.random(m * n) < 0.5] *= -1.0
    q = np.ones((m, n, 4))
    q[..., 0], q[..., 1], q[..., 2] = rho.reshape(m, n), num.reshape(m, n), num[::-1].reshape(m, n)
    wx.set_mode("exact")
    _, _, r, u, v, _ = wx.con2primi_py(q, 1.4)
    assert np.array_equal(r, q[..., 0])
    with np.errstate(all="ignore"):
        assert np.array_equal(u.view(np.uint64), (q[..., 1] / q[..., 0]).view(np.uint64))
        assert np.array_equal(v.view(np.uint64), (q[..., 2] / q[..., 0]).view(np.uint64))
