"""Objectives of a few forward steps, around the number up to which they take their
own way to the host (a handle's page, a batch's objective kernels): each step's
value, a handle's sum and a batch's, against the oracle."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,tol", [(G.STORE_FP64, 1e-12), (G.STORE_FP32, 1e-5)])
@pytest.mark.parametrize("objective", [G.OBJ_PRESSURE_DROP, G.OBJ_DISSIPATION])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6])
def test_few_steps(orc, n, objective, storage, tol):
    cfgs = [W.channel_2d(nx, ny, nsteps=1, objective=objective, storage=storage)
            for nx, ny in ((41, 20), (70, 33))]
    gs = [W.design_2d(c.nx, c.ny, 5) for c in cfgs]
    rng = np.random.default_rng(2)
    macs = []
    for c in cfgs:
        m = np.zeros((c.ncells, 3))
        m[:, 0] = 1 + 0.02 * rng.uniform(-1, 1, c.ncells)
        m[:, 1:] = 0.04 * rng.uniform(-1, 1, (c.ncells, 2))
        macs.append(m.ravel())
    want = [orc.forward(c.replace(storage=G.STORE_FP64), g, n, macros=m)[1]
            for c, g, m in zip(cfgs, gs, macs)]
    size = [np.abs(j).max() for j in want]
    with G.Batch(cfgs) as b:
        for i in range(2):
            b[i].set_design(gs[i])
            b[i].init_equilibrium(macs[i])
        Jb = b.forward(n)
    for i, c in enumerate(cfgs):
        with G.Handle(c) as h:
            h.set_design(gs[i])
            h.init_equilibrium(macs[i])
            J, js = h.forward(n, per_step=True)
            h.init_equilibrium(macs[i])
            Js = h.forward(n)
        assert js.shape == (n,) and np.abs(js - want[i]).max() <= tol * size[i]
        for v in (J, Js, Jb[i]):
            assert abs(v - want[i].sum()) <= tol * size[i] * n
