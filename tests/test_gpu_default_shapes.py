"""Default block shapes and launch overlap of the step kernels by lattice size:
on both sides of each line of the rules (half a block per SM, two and four
blocks of 256 threads, one wave of forward blocks on 152 SMs, the grid's limit
along y), populations and sensitivities are the bits of one fixed shape."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu

CASES = [(5, 3), (64, 48), (256, 76), (256, 77), (255, 97), (201, 201), (256, 304), (256, 305),
         (256, 608), (250, 609), (512, 456), (512, 457), (32, 70000)]


def results(cfg, gamma, n, shape=None):
    with G.Handle(cfg) as h:
        if shape:
            h.set_launch_shape(0, *shape)
            h.set_launch_shape(1, *shape)
        h.set_design(gamma)
        h.init_equilibrium()
        J, s, _ = h.gradient(n, 2)
        h.init_equilibrium()
        h.forward(n)
        return J, s, h.populations()


@pytest.mark.parametrize("storage", [G.STORE_FP64, G.STORE_FP32, G.STORE_FP16])
@pytest.mark.parametrize("nx,ny", CASES)
def test_2d_bits(nx, ny, storage):
    n = 7
    cfg = W.channel_2d(nx, ny, storage=storage, nsteps=n)
    gamma = W.design_2d(nx, ny, 4)
    J, s, f = results(cfg, gamma, n)
    J1, s1, f1 = results(cfg, gamma, n, (32, 8) if ny > 1000 else (256, 1))
    assert np.array_equal(f, f1) and np.array_equal(s, s1)
    # the step sums add the warps' shares, each at most 1/n in all, in another order
    assert abs(J - J1) <= 1e-12


@pytest.mark.parametrize("storage", [G.STORE_FP64, G.STORE_FP32, G.STORE_FP16])
@pytest.mark.parametrize("dims", [(3, 3, 3), (32, 16, 16), (33, 17, 38), (70, 20, 40), (64, 64, 41), (96, 63, 41),
                                  (97, 63, 41)])
def test_3d_bits(dims, storage):
    n = 5
    cfg = W.duct_3d(*dims, storage=storage, nsteps=n)
    gamma = W.design_3d(*dims, 4)
    J, s, f = results(cfg, gamma, n)
    J1, s1, f1 = results(cfg, gamma, n, (256, 1))
    assert np.array_equal(f, f1) and np.array_equal(s, s1)
    assert abs(J - J1) <= 1e-12
