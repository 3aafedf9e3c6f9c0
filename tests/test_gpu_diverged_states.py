"""FP64 reverse steps at states that have diverged in a cell, where no adjoint has
arrived: zero times what is not finite is not a number, in the adjoint and in
dJ/dgamma, as with the FP64 operators (here the oracle's)."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def config(name):
    if name.startswith("d3q19"):
        return W.duct_3d(13, 11, 9).replace(collision=G.BGK if name.endswith("bgk") else G.MRT)
    if name == "thermal":
        return W.thermal_2d(24, 17).replace(objective=G.OBJ_DOMAIN_TEMPERATURE,
                                            obj_out=(2, 3, 2, 3, 0, 0))
    return W.channel_2d(24, 17, collision=G.BGK if name.endswith("bgk") else G.MRT,
                        objective=G.OBJ_PRESSURE_DROP)


# (whether the squares of 1e160 and more meet the zeros is a matter of the operators' form)
VALUES = [np.nan, np.inf, -np.inf, 1e100, 1e3, -0.05, 0.0, 5e-324]


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("name", ["d2q9_bgk", "d2q9_mrt", "d3q19_mrt", "d3q19_bgk", "thermal"])
def test_zero_adjoint_at_a_diverged_cell(orc, name, whole):
    cfg = config(name)
    q, z = cfg.npop, cfg.nz // 2
    cell = (z * cfg.ny + cfg.ny // 2) * cfg.nx + cfg.nx // 2
    gamma = np.full(cfg.ncells, 0.5)
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        h.init_equilibrium()
        f0 = h.populations().reshape(-1, q)
        for v in VALUES:
            # (the rest population has no part in the momentum, which is all that
            # the transposes need of a state)
            for k in ([None] if whole else range(1, q)):
                f = f0.copy()
                if whole:
                    f[cell] = v
                else:
                    f[cell, k] = v
                lam, dg = orc.reverse_cell(cfg, f[cell], 0.5, np.zeros(q))
                h.set_populations(f, 3)
                h.adjoint_reset()
                h.adjoint_step()
                s, a = h.sensitivity(), h.adjoint()
                assert np.isfinite(s[cell]) == np.isfinite(dg), (v, k)
                # (so is which components)
                assert np.isfinite(a).all() == np.isfinite(lam).all(), (v, k)
                assert np.isfinite(np.delete(s, cell)).all()
