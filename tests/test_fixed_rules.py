"""Which models of FP64 storage run their collisions in fixed point
(fixed_model.hpp), seen through the host build.  Runs without a GPU."""
import pytest

import workloads as W
from test_fixed_math_host import lib, run_forward, states  # noqa: F401  (lib: fixture)


def taken(lib, cfg):
    f, g = states(cfg, 100, 3, 0.02)
    return run_forward(lib, cfg, f, g)[0]


@pytest.mark.parametrize("n", [12, 36, 60, 201])
def test_velocity_objectives_do_not_depend_on_the_size(lib, n):
    assert taken(lib, W.pump_2d(n)) == 100
