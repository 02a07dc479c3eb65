"""Both sides of each line of the four-lanes-per-face rule (csrc/launch_api.h: 14, 16 or 24 blocks of eight faces
per SM): the residual and the reconstruction against the oracle, bit for bit in exact mode and within the
one-call tolerance in fast mode, and the solver's steps on a grid next to each line."""

import numpy as np
import pytest

from states import quadrant
from test_gpu_dropin import check, mode  # noqa: F401
from test_gpu_solver import oracle_run

pytestmark = pytest.mark.gpu
G = 1.4
# faces per sweep just below and just above 17,024, 19,456 and 29,184, and a thin array around 19,456
SHAPES = [(132, 133), (133, 134), (142, 141), (142, 143), (173, 173), (174, 174), (12, 1626), (12, 1628)]


@pytest.mark.parametrize("mn", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("cons", [True, False], ids=["cons", "char"])
@pytest.mark.parametrize("hlle", [True, False], ids=["hlle", "blend"])
def test_residual(wx, orc, mode, mn, cons, hlle):  # noqa: F811
    rng = np.random.default_rng(sum(mn))
    q = quadrant(rng, mn[0] - 6, mn[1] - 6)
    q[..., :4] *= 1.0 + 0.01 * rng.random(q.shape[:2])[..., None]
    args = (0.01, G, hlle, (0.2, 1.0), cons)
    check(wx.l_local_py(q, *args), orc.l_local_py(q, *args), mode)


@pytest.mark.parametrize("mn", SHAPES[2:], ids=lambda s: f"{s[0]}x{s[1]}")
def test_reconstruct(wx, orc, mode, mn):  # noqa: F811
    q = quadrant(np.random.default_rng(sum(mn)), mn[0] - 6, mn[1] - 6)
    for cons in (True, False):
        for fw, fo in ((wx.weno_x_py, orc.weno_x_py), (wx.weno_y_py, orc.weno_y_py)):
            for got, ref in zip(fw(q, G, cons=cons), fo(q, G, cons=cons)):
                check(got, ref, mode)


@pytest.mark.parametrize("mn,hlle,quads", [((132, 133), False, True), ((133, 134), False, False),
                                           ((142, 141), True, True), ((142, 143), True, False)])
def test_solver(wx, orc, mn, hlle, quads):
    """Exact steps, and as many launches as the rule says: two fewer per residual below the line."""
    nx, ny = mn[0] - 6, mn[1] - 6
    q = orc.bc_transmissive(quadrant(np.random.default_rng(3), nx, ny))
    ref = oracle_run(orc, q.copy(), nx, ny, 1 / ny, 0.4, 2, jp=(0.05, 0.4), hlle=hlle)[0]
    s = wx.Solver(nx, ny, 1 / ny, G, mode="exact", force_hlle=hlle, jp_cri=(0.05, 0.4), cfl=0.4)
    s.set_state(q)
    s.run(2)
    check(s.state(), ref, "exact")
    assert s.launches_per_step == 4 + 3 * (5 + (0 if hlle else 2) - (2 if quads else 0) + 1)
