"""The design kernels at the sizes where their blocks and reductions can go
wrong, against the CPU oracle: filters on grids around the 64 x 4 blocks,
narrower than a tap's reach and with filter boxes thinner than it (every cell
takes the tested path) or much larger (most take the untested one), and MMA at
every number of constraints and at sizes around the blocks and the resident
grid of its reductions.  Tolerances as in test_gpu_design.py: 1e-13 for the
filters, 1e-10 for MMA."""
import numpy as np
import pytest

import design_lib as D
import lbmgpu as G
from test_gpu_design import box_mask

pytestmark = pytest.mark.gpu

FILTERS = [
    (63, 3, 1, (0, 62, 0, 2, 0, 0), 4),
    (64, 4, 1, (1, 62, 1, 2, 0, 0), 1),
    (65, 5, 1, (2, 62, 0, 4, 0, 0), 3),
    (200, 37, 1, (3, 190, 2, 33, 0, 0), 9),
    (5, 300, 1, (0, 4, 10, 280, 0, 0), 2),
    (66, 9, 7, (4, 60, 1, 7, 1, 5), 3),
    (12, 11, 30, (1, 10, 1, 9, 2, 27), 2),
]


@pytest.mark.parametrize("nx,ny,nz,box,radius", FILTERS)
def test_filter_blocks(nx, ny, nz, box, radius):
    rng = np.random.default_rng(nx * ny + radius)
    N = nx * ny * nz
    bg, s = rng.uniform(0, 1, N), rng.standard_normal(N)
    mask = box_mask(nx, ny, nz, box)
    x = rng.uniform(0, 1, int(mask.sum()))
    stages = [(radius, True, 2.0, 0.4), (max(1, radius - 1), True, 5.0, 0.6)]
    with G.TopOpt(nx, ny, nz, box, stages, background=bg, x0=x) as t:
        gam = t.physical(0)
        t.set_sensitivity_host(0, s, 1.0)
        dx = t.design_sensitivity(0)
    ch = D.make_chain(nx, ny, nz, [(r, box, p, b, e) for r, p, b, e in stages])
    xfull = bg.copy()
    xfull[mask] = x
    assert np.abs(gam - D.filter_forward(ch, xfull)).max() <= 1e-13
    dx_o = D.filter_transpose(ch, xfull, s)[mask]
    assert np.abs(dx - dx_o).max() <= 1e-13 * max(1.0, np.abs(dx_o).max())


MMA = [(1, 255), (2, 256), (3, 257), (4, 31), (5, 300), (6, 1000), (7, 511), (8, 513),
       (3, 77823), (4, 77825), (1, 160001)]


@pytest.mark.parametrize("nreal,n", MMA)
def test_mma_constraint_counts_and_sizes(nreal, n):
    """min-max of nreal quadratics with a volume constraint (nreal = 1: one
    quadratic, one constraint), five updates."""
    rng = np.random.default_rng(100 * nreal + n)
    t = rng.uniform(0, 1, (nreal, n))
    w = rng.uniform(0.5, 2, (nreal, n))
    m = 1 if nreal == 1 else nreal + 1
    a = None if nreal == 1 else np.array([1.0] * nreal + [0.0])
    x = np.full(n, 0.5)
    orc, xo = D.OracleMMA(n, m, x, a), x.copy()

    def ev(x):
        J = [np.sum(w[k] * (x - t[k]) ** 2) / n for k in range(nreal)]
        return J, [2 * w[k] * (x - t[k]) / n for k in range(nreal)]

    with G.TopOpt(n, 1, 1, (0, n - 1, 0, 0, 0, 0), stages=(), nreal=nreal, volume=0.45,
                  move_limit=0.1, magic=5.0, x0=x) as top:
        for _ in range(5):
            J, dJ = ev(x)
            for r in range(nreal):
                top.set_sensitivity_host(r, dJ[r], J[r])
            ch, _ = top.update()
            x = top.variables()
            J, dJ = ev(xo)
            vol = np.full(n, 1.0 / n)
            if nreal == 1:
                df0, g, dg = dJ[0], np.array([xo.mean() - 0.45]), vol[None]
            else:
                df0, g = np.zeros(n), np.array([v + 5 for v in J] + [xo.mean() - 0.45])
                dg = np.vstack(dJ + [vol])
            xo, cho, _ = orc.update(xo, df0, g, dg, 0.1)
            assert np.abs(x - xo).max() < 1e-10
            assert abs(ch - cho) < 1e-10
