"""FP64 storage with a velocity objective: the first steps keep the FP64
operators (flow_start_up in fixed_model.hpp).  Which operators a step runs is a
matter of the model and of the step's time alone: not of how a sweep is cut into
calls, nor of what the handle did before."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu

N = 60   # sound takes 49 steps to the outlets


def pump(h, cfg):
    h.set_bc_profile(2, W.pump_inflow_profile(cfg))
    h.set_design(W.design_2d(N, N, 9))


def config(collision=G.MRT):
    return W.pump_2d(N, collision=collision, nsteps=200, period=100.0)


@pytest.mark.parametrize("collision", [G.BGK, G.MRT])
@pytest.mark.parametrize("cuts", [[50] * 4, [1] * 200, [83, 1, 1, 115], [180, 20]])
def test_sweep_cut_into_calls_gives_the_same_bits(collision, cuts):
    cfg = config(collision)
    with G.Handle(cfg) as h:
        pump(h, cfg)
        h.init_equilibrium()
        _, whole = h.forward(200, per_step=True)
        f = h.populations()
        h.init_equilibrium()
        parts = np.concatenate([h.forward(n, per_step=True)[1] for n in cuts])
        assert np.array_equal(h.populations(), f)
    assert np.array_equal(parts, whole)


@pytest.mark.parametrize("t", [40, 120])
def test_adjoint_step_does_not_depend_on_earlier_sweeps(t):
    cfg = config()
    rng = np.random.default_rng(1)
    with G.Handle(cfg) as h:
        pump(h, cfg)
        h.init_equilibrium()
        h.forward(t)
        f = h.populations() * (1 + 1e-6 * rng.standard_normal(cfg.ncells * 9))

    def reverse(h):
        h.adjoint_reset()
        for k in range(3):
            h.set_populations(f, t - k)
            h.adjoint_step()
        return h.adjoint(), h.sensitivity()

    with G.Handle(cfg) as h:
        pump(h, cfg)
        fresh = reverse(h)
    with G.Handle(cfg) as h:
        pump(h, cfg)
        h.init_equilibrium()
        h.forward(250)
        after = reverse(h)
        h.time_steps(2, 3)
        h.set_populations(f, t)
        h.autotune(1)
        tuned = reverse(h)
    with G.Batch([cfg, cfg]) as b:
        for k in range(2):
            pump(b[k], cfg)
        b.autotune(1)
        b.time_steps(0, 2)
        batched = reverse(b[1])
    for other in (after, tuned, batched):
        assert np.array_equal(other[0], fresh[0])
        assert np.array_equal(other[1], fresh[1])


@pytest.mark.parametrize("n", [80, 90, 110, 180])
def test_sweeps_that_end_around_the_change(orc, n):
    """J and dJ/dgamma against the FP64 oracle.  Each step's velocities, averaged
    over the outlets, carry a rounding of some 5e-17 of the weight (1 / 200)."""
    cfg = config()
    gamma, table = W.design_2d(N, N, 9), W.pump_inflow_profile(cfg)
    with G.Handle(cfg) as h:
        pump(h, cfg)
        h.init_equilibrium()
        _, js = h.forward(n, per_step=True)
        J, s, _ = h.gradient(n, 10)
    try:
        orc.set_tables({2: table})
        _, jo, _ = orc.forward(cfg, gamma, n)
        Jo, so = orc.gradient(cfg, gamma, n)
    finally:
        orc.set_tables()
    drift = 5e-17 * n
    assert np.abs(js - jo).max() < drift / 200 * 4 and abs(J - Jo) < drift
    assert np.abs(s - so).max() <= 1e-12 * np.abs(so).max() + drift / 200
