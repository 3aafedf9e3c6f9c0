"""The filter kernels where a warp's cells (32 of a row, from a multiple of 32 on)
have all, some or none of their taps inside the field and the filter box: rows and
boxes around those lines, against the CPU oracle.  Tolerance as in
test_gpu_design.py: 1e-13 for the filters."""
import numpy as np
import pytest

import design_lib as D
import lbmgpu as G
from test_gpu_design import box_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1, 2, 4, 9])
@pytest.mark.parametrize("x0,x1", [(0, 0), (1, 1), (3, 2), (32, 0), (0, 33), (31, 31)])
@pytest.mark.parametrize("nx,ny,nz", [(31, 23, 1), (32, 23, 1), (34, 9, 8), (65, 22, 1), (98, 20, 1),
                                      (112, 21, 1)])
def test_rows_and_boxes(nx, ny, nz, x0, x1, radius):
    """Filter boxes that leave out x0 cells on the left and x1 on the right."""
    if x0 + x1 >= nx or (nz > 1 and radius > 4):
        pytest.skip("no cell left, or many taps")
    box = (x0, nx - 1 - x1, 1, ny - 2, 1 if nz > 1 else 0, nz - 2 if nz > 1 else 0)
    rng = np.random.default_rng(nx + 7 * radius + x0)
    N = nx * ny * nz
    bg, s = rng.uniform(0, 1, N), rng.standard_normal(N)
    mask = box_mask(nx, ny, nz, box)
    x = rng.uniform(0, 1, int(mask.sum()))
    with G.TopOpt(nx, ny, nz, box, [(radius, True, 2.0, 0.4)], background=bg, x0=x) as t:
        gam = t.physical(0)
        t.set_sensitivity_host(0, s, 1.0)
        dx = t.design_sensitivity(0)
    ch = D.make_chain(nx, ny, nz, [(radius, box, True, 2.0, 0.4)])
    xfull = bg.copy()
    xfull[mask] = x
    assert np.abs(gam - D.filter_forward(ch, xfull)).max() <= 1e-13
    dx_o = D.filter_transpose(ch, xfull, s)[mask]
    assert np.abs(dx - dx_o).max() <= 1e-13 * max(1.0, np.abs(dx_o).max())
