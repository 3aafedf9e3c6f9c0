"""The two register budgets of the FP64 D2Q9 reverse step (chosen by the number of
cells, or by the tuners): the same results, and one variant for the caller."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu

N = 12
# a cell's share of dJ/dgamma is a sum of doubles that the compiler may fuse
# differently: some four roundings of it in each of the N + 1 steps
TOL = 4 * (N + 1) * 2.0 ** -53


def config(nx, ny, collision, objective):
    return W.channel_2d(nx, ny, nsteps=N, collision=collision, objective=objective, amp=0.2,
                        period=9.0)


@pytest.mark.parametrize("objective", [G.OBJ_PRESSURE_DROP, G.OBJ_DISSIPATION])
@pytest.mark.parametrize("collision", [G.BGK, G.MRT])
@pytest.mark.parametrize("nx,ny", [(304, 256), (305, 256), (97, 81)])
def test_budgets_agree(collision, objective, nx, ny):
    """152 SMs: 304x256 cells are the last to run alone with the larger budget;
    beside a 320x280 lattice all run with the smaller one."""
    cfg, big = config(nx, ny, collision, objective), config(320, 280, collision, objective)
    g = W.design_2d(nx, ny, 6)
    with G.Handle(cfg) as h:
        h.set_design(g)
        J, s, _ = h.gradient(N, 4)
        h.init_equilibrium()
        h.autotune(1)
        Jt, st, _ = h.gradient(N, 4)
    with G.Batch([big, cfg]) as b:
        b[0].set_design(W.design_2d(320, 280, 7))
        b[1].set_design(g)
        Jb, sb, _ = b.gradient(N, 4)
    for Jo, so in ((Jt, st), (Jb[1], sb[1])):
        assert abs(Jo - J) <= 1e-13 * abs(J)
        assert np.abs(so - s).max() <= TOL * np.abs(s).max()


@pytest.mark.parametrize("nx,ny", [(96, 40), (320, 280)])
def test_fp64_has_one_variant_for_the_caller(nx, ny):
    cfg = config(nx, ny, G.BGK, G.OBJ_PRESSURE_DROP)
    with G.Handle(cfg) as h, G.Batch([cfg]) as b:
        h.set_design(W.design_2d(nx, ny, 6))
        h.init_equilibrium()
        b[0].set_design(W.design_2d(nx, ny, 6))
        for o in (h, b):
            for tune in (False, True):
                if tune:
                    o.autotune(1)
                assert o.reverse_variant == 0
                o.set_reverse_variant(0)
                assert o.reverse_variant == 0
                with pytest.raises(G.LBMError) as e:
                    o.set_reverse_variant(1)
                assert e.value.code == G.ERR_SUP
