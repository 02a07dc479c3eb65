"""The kernel classes of the timing report (include/weno_gb300.h): every class that a configuration runs has its
launch groups, on small FP64 grids too, whose sweeps otherwise share their launches; timing changes no result."""

import ctypes

import numpy as np
import pytest

from states import quadrant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [24, 180])
@pytest.mark.parametrize("precision,mode", [(64, "exact"), (64, "fast"), ("df64", "fast"), (32, "fast")])
@pytest.mark.parametrize("hlle", [True, False], ids=["hlle", "blend"])
def test_classes(wx, n, precision, mode, hlle):
    from weno_ext import _lib
    L = _lib.load()
    q = quadrant(np.random.default_rng(5), n, n)
    states = []
    for timing in (0, 1):
        s = wx.Solver(n, n, 1 / n, precision=precision, mode=mode, force_hlle=hlle, cfl=0.4)
        s.set_state(q)
        _lib.check(L.weno_solver_enable_timing(s._h, timing), "timing")
        s.run(2, graph=False)
        states.append(s.state())
        if timing:
            ms, groups = (ctypes.c_double * 8)(), (ctypes.c_int64 * 8)()
            _lib.check(L.weno_solver_timing_report(s._h, ms, groups, 8), "report")
        s.close()
    assert np.array_equal(states[0], states[1], equal_nan=True)
    blends = 0 if hlle or precision == 32 else 2 * 6
    assert list(groups) == [2, 8, 6, 6, blends, 6, 6, 6]
    assert all((t > 0) == (g > 0) for t, g in zip(ms, groups))
