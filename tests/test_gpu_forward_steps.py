"""lbm_forward's objective of every step, of a sweep and of single steps: the
same values along the three paths (rows of partial sums, sums over the sweep,
the objective kernel alone), at step counts around the 64 rows kept at a time
and on a lattice whose rows are so long that fewer are kept."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W
from helpers import rel_inf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 66, 129])
@pytest.mark.parametrize("objective", [G.OBJ_PRESSURE_DROP, G.OBJ_DISSIPATION])
def test_steps_and_sums_match_the_oracle(orc, objective, n):
    cfg = W.channel_2d(27, 14, nsteps=n, amp=0.2, period=11.0, objective=objective)
    gamma = W.design_2d(27, 14, 3)
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        h.init_equilibrium()
        J, js = h.forward(n, per_step=True)
        h.init_equilibrium()
        total = h.forward(n)
        h.init_equilibrium()
        single = np.array([h.forward(1) for _ in range(n)])
    _, jo, Jo = orc.forward(cfg, gamma, n)
    assert rel_inf(js, jo) < 1e-12 and rel_inf(single, jo) < 1e-12
    assert abs(J - Jo) <= 1e-12 * np.abs(jo).sum() and abs(total - Jo) <= 1e-12 * np.abs(jo).sum()


@pytest.mark.parametrize("storage", [G.STORE_FP64, G.STORE_FP32, G.STORE_FP16])
def test_long_rows(storage):
    """2048x1100: rows of 70,400 partial sums and more, at most 59 of them kept;
    single steps take the summed path.  FP64 sums of the same warps' values."""
    n = 61
    cfg = W.channel_2d(2048, 1100, storage=storage, nsteps=n, objective=G.OBJ_DISSIPATION)
    with G.Handle(cfg) as h:
        h.set_design(W.design_2d(2048, 1100, 5))
        h.init_equilibrium()
        J, js = h.forward(n, per_step=True)
        h.init_equilibrium()
        single = np.array([h.forward(1) for _ in range(n)])
        h.init_equilibrium()
        total = h.forward(n)
    assert rel_inf(js, single) < 1e-13
    assert abs(J - total) <= 1e-13 * np.abs(js).sum()
