"""MMA steps with derivatives that are not numbers: a constraint's derivative enters
as max(0, g) and max(0, -g), which such a value leaves at zero."""
import numpy as np
import pytest

import lbmgpu as G

pytestmark = pytest.mark.gpu


def update(nreal, s, steps=2):
    nx, ny = 40, 24
    with G.TopOpt(nx, ny, 1, (0, nx - 1, 0, ny - 1, 0, 0), stages=[], nreal=nreal,
                  volume_type=G.VOLUME_FLUID, volume=0.6, x0=np.full(nx * ny, 0.5)) as t:
        for _ in range(steps):
            for r in range(nreal):
                t.set_sensitivity_host(r, s[r], 0.1 + 0.01 * r)
            change, cons = t.update()
        return change, np.asarray(cons), t.variables()


@pytest.mark.parametrize("nreal", [2, 5, 8])
def test_not_a_number_counts_as_zero(nreal):
    rng = np.random.default_rng(3)
    zero = [1e-6 * rng.standard_normal(40 * 24) for _ in range(nreal)]
    nan = [s.copy() for s in zero]
    for r in range(nreal):
        zero[r][r::97] = 0.0
        nan[r][r::97] = np.nan
    a, b = update(nreal, zero), update(nreal, nan)
    assert np.isfinite(a[0]) and a[0] == b[0]
    assert np.array_equal(a[1], b[1])
    assert np.isfinite(a[2]).all() and np.array_equal(a[2], b[2])
