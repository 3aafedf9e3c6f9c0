"""FP64 storage on the GPU, whose collisions run in fixed point where a cell's
populations allow it (lbm_fixed.cuh), against the oracle on lattices whose
cells lie inside, outside and across the accepted range (velocities and
densities to both sides of its limits), and with designs that the porosity
plane does not hold.  Tolerance 1e-12 as for every FP64 comparison."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W
from helpers import rel_inf

pytestmark = pytest.mark.gpu

TOL = 1e-12


def config(name):
    if name == "d3q19_mrt":
        return W.duct_3d(13, 9, 7, nsteps=12), W.design_3d(13, 9, 7, 3)
    if name == "d2q9_bgk":
        return W.channel_2d(21, 14, nsteps=12, amp=0.2, period=9.0), W.design_2d(21, 14, 3)
    if name == "d2q9_mrt":
        return W.channel_2d(33, 9, nsteps=12, collision=G.MRT), W.design_2d(33, 9, 4)
    if name == "d2q9_bgk_dissipation":
        return (W.channel_2d(40, 23, nsteps=12, objective=G.OBJ_DISSIPATION, amp=0.2, period=9.0),
                W.design_2d(40, 23, 5))
    if name == "d3q19_bgk":
        return W.duct_3d(9, 11, 6, nsteps=12).replace(collision=G.BGK), W.design_3d(9, 11, 6, 6)
    if name == "thermal":
        return W.thermal_2d(35, 18, nsteps=12, period=9.0), W.thermal_design(35, 18, 7)
    if name == "regenerator":
        return (W.regenerator_2d(30, 17, n_unsteady=12, objective=G.OBJ_DOMAIN_TEMPERATURE),
                W.regenerator_design(30, 17, 8))
    raise KeyError(name)


def macros(cfg, drho, u, seed):
    rng = np.random.default_rng(seed)
    m = np.zeros((cfg.ncells, cfg.nmac))
    m[:, 0] = 1 + drho * rng.uniform(-1, 1, cfg.ncells)
    dim = 3 if cfg.lattice == G.D3Q19 else 2
    m[:, 1:1 + dim] = u * rng.uniform(-1, 1, (cfg.ncells, dim))
    if cfg.lattice == G.D2Q9_D2Q5:
        m[:, 3] = rng.uniform(0, 1, cfg.ncells)
    return m.ravel()


MODELS = ["d3q19_mrt", "d2q9_bgk", "d2q9_mrt", "d2q9_bgk_dissipation", "d3q19_bgk", "thermal",
          "regenerator"]


@pytest.mark.parametrize("drho,u", [(0.0, 0.02), (0.15, 0.1), (0.6, 0.3)])
@pytest.mark.parametrize("name", MODELS)
def test_inside_across_and_outside_the_range(orc, name, drho, u):
    cfg, gamma = config(name)
    mac = macros(cfg, drho, u, 5)
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        h.init_equilibrium(mac)
        J, js = h.forward(12, per_step=True)
        f = h.populations()
        Jg, s, _ = h.gradient(12, 3)
    fo, jo, _ = orc.forward(cfg, gamma, 12, macros=mac)
    assert rel_inf(f, fo) < TOL
    assert rel_inf(js, jo) < TOL
    Jo, so = orc.gradient(cfg, gamma, 12, macros=mac)
    assert abs(Jg - Jo) <= TOL * abs(jo).max() * 12
    assert rel_inf(s, so) < TOL


@pytest.mark.parametrize("name", MODELS)
def test_large_drag_leaves_the_porosity_plane(orc, name):
    """interp_scale = 1.6: imult up to 0.8, outside the plane's [0, 1/2]."""
    cfg, gamma = config(name)
    cfg = cfg.replace(interp_scale=1.6)
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        h.init_equilibrium()
        h.forward(12)
        f = h.populations()
    fo, _, _ = orc.forward(cfg, gamma, 12)
    assert rel_inf(f, fo) < TOL


@pytest.mark.parametrize("n", [60, 420])
def test_velocity_objective_before_and_after_the_flow_arrives(orc, n):
    """75x75 pump: the pressure wave takes some 60 steps to the outlets.  Sweeps
    up to 194 steps keep the FP64 operators, longer ones do not."""
    cfg = W.pump_2d(75, nsteps=n, period=100.0)
    gamma, table = W.design_2d(75, 75, 9), W.pump_inflow_profile(cfg)
    with G.Handle(cfg) as h:
        h.set_bc_profile(2, table)
        h.set_design(gamma)
        h.init_equilibrium()
        J, js = h.forward(n, per_step=True)
        Jg, s, _ = h.gradient(n, 10)
    try:
        orc.set_tables({2: table})
        _, jo, _ = orc.forward(cfg, gamma, n)
        Jgo, so = orc.gradient(cfg, gamma, n)
    finally:
        orc.set_tables()
    # the FP64 velocities drift by about 2e-17 a step
    drift = 5e-17 * n
    assert np.abs(js - jo).max() < drift / n and abs(Jg - Jgo) < drift
    assert np.abs(s - so).max() <= 1e-12 * np.abs(so).max() + drift / n


@pytest.mark.parametrize("objective,box", [
    (G.OBJ_DISSIPATION, None),
    (G.OBJ_PRESSURE_DROP, (0, 0, 1, 38, 0, 0)),      # one lane of a warp
    (G.OBJ_PRESSURE_DROP, (0, 40, 7, 7, 0, 0)),      # a full warp and a part of one
    (G.OBJ_PRESSURE_DROP, (31, 32, 3, 3, 0, 0)),     # one lane each of two warps
])
@pytest.mark.parametrize("amp", [0.0, 1e-7, 0.05])
def test_sums_over_the_warp(orc, objective, box, amp):
    """Objectives that all, some or single lanes of a warp contribute to, from a
    fluid at rest, a slow and a fast flow; J of a sweep and of its steps."""
    nx, ny, n = 41, 40, 9
    cfg = W.channel_2d(nx, ny, nsteps=n, objective=objective)
    if box:
        cfg = cfg.replace(obj_in=box)
    gamma = W.design_2d(nx, ny, 5)
    mac = np.zeros((nx * ny, 3))
    mac[:, 0] = 1.0
    mac[:, 1:] = amp * np.random.default_rng(3).uniform(-1, 1, (nx * ny, 2))
    with G.Handle(cfg) as h:
        h.set_design(gamma)
        h.init_equilibrium(mac)
        _, js = h.forward(n, per_step=True)
        h.init_equilibrium(mac)
        J, _, _ = h.gradient(n, 3)
    _, jo, _ = orc.forward(cfg, gamma, n, macros=mac)
    # a step's J adds up to nx ny values of the size of its largest cell's, whose
    # own roundings are a few 2^-53 of a density (pressure) or of j^2 and V^2
    size = np.abs(jo).max() if objective == G.OBJ_DISSIPATION else 1.0 / n
    assert np.abs(js - jo).max() <= 1e-13 * size
    assert abs(J - jo.sum()) <= 1e-13 * size * n


@pytest.mark.parametrize("collision", [G.BGK, G.MRT])
def test_dissipation_adjoint_of_a_fluid_at_rest(collision):
    """Cells that the flow has not reached: every product of the source and of
    the transposed collision has a zero operand, and the adjoint has to stay
    within the units of 2^-61 of the weight that the products may lose (some
    tens of them a step; a lost carry is 2^32 of them)."""
    nx, ny, n = 160, 40, 4
    cfg = W.channel_2d(nx, ny, nsteps=n, objective=G.OBJ_DISSIPATION, collision=collision)
    with G.Handle(cfg) as h:
        h.set_design(W.design_2d(nx, ny, 6))
        h.init_equilibrium()
        states = []
        for t in range(1, n + 1):
            h.forward(1)
            states.append(h.populations())
        h.adjoint_reset()
        for t in range(n, 0, -1):
            h.set_populations(states[t - 1], t)
            h.adjoint_step()
        lam = h.adjoint().reshape(ny, nx, 9)
    far = lam[8:-8, 20:-20]
    assert np.abs(far).max() <= 1000 * n * 2.0 ** -61 * abs(cfg.obj_weight)
    assert np.abs(lam).max() > 1e-9 * abs(cfg.obj_weight)
