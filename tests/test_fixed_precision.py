"""The fixed-point forms of FP64 storage (lbm_fixed.cuh) against extended precision
beyond single collisions: sweeps of the flow and temperature lattices, whole reverse
steps with the dissipation source from slow and fast flows, and weak porosity.
Runs without a GPU."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import lbmgpu as G
import workloads as W
from test_device_math_host import _cuda_include
from test_fixed_math_host import (E2, E5, LD, W2, W5, collide_exact, lib, model,  # noqa: F401
                                  ptr, reverse_exact, run_forward, states)

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def source_lib(tmp_path_factory):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    so = str(tmp_path_factory.mktemp("src") / "libfixedsource.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-ffp-contract=off",
                           "-I" + inc, os.path.join(HERE, "fixed_source_host.cpp"), "-o", so])
    return C.CDLL(so)


def imult_of(cfg, g):
    """The design's porosity factor, a double that both forms take."""
    q = cfg.interp_q
    return (0.5 * (cfg.interp_scale * (1.0 - g * (1.0 + q) / (q + g)))).astype(LD)


def rms(v):
    return float(np.sqrt((v.astype(LD) ** 2).mean()))


def streamed(a, E, nx, ny, sign=1):
    v = a.reshape(ny, nx, -1)
    out = [np.roll(v[..., q], (sign * int(E[q][1]), sign * int(E[q][0])), (0, 1))
           for q in range(len(E))]
    return np.ascontiguousarray(np.stack(out, -1).reshape(a.shape))


@pytest.mark.parametrize("solid", [False, True])
@pytest.mark.parametrize("tau", [0.8, 0.6])
def test_thermal_sweep(lib, tau, solid):  # noqa: F811
    """300 steps of flow and temperature on a periodic lattice, then the temperature's
    adjoint back over the recorded flow: within the FP64 operators' error, which is a
    drift, 20 times over (the fixed form's error is that of one rounding)."""
    nx, ny, steps = 20, 14, 300
    n, rng = nx * ny, np.random.default_rng(4)
    cfg = W.thermal_2d(nx, ny, tau=tau, heat_rate=0.0).replace(objective=G.OBJ_PRESSURE_DROP)
    flow = cfg.replace(lattice=G.D2Q9)
    c = flow.to_c()
    f, _ = states(model("d2q9_bgk"), n, 4, 0.03)
    g = rng.uniform(0, 1, n) if solid else np.ones(n)
    t = np.ascontiguousarray(W5.astype(float) * rng.uniform(0.2, 1, (n, 1)) *
                             (1 + 0.05 * rng.standard_normal((n, 5))))
    q, ck = cfg.ramp_q, cfg.ramp_ck
    om = 1 / (3 * cfg.diffusivity * (g * (ck * (1 + q) - 1) + 1) / (ck * (1 + q * g)) + 0.5)
    im, omL = imult_of(cfg, g), om.astype(LD)[:, None]

    def step(f, t, l):
        a, b = np.empty((n, 9)), np.empty((n, 9))
        o = [np.zeros((n, 5)) for _ in range(4)]
        misc = np.zeros((n, 3))
        assert lib.fixed_forward(C.byref(c), n, ptr(f), ptr(g), ptr(a), ptr(b)) == n
        assert lib.fixed_thermal(n, ptr(f), ptr(t), ptr(l), ptr(om), *[ptr(v) for v in o],
                                 ptr(misc)) == n
        return (a, o[0], o[2]), (b, o[1], o[3])

    def geq(f):
        j = (f @ E2.astype(LD))[:, :2]
        return W5 * (1 + 3 * (j @ E5.T.astype(LD)))

    fixed, fp64, ref = (f, t), (f, t), (f.astype(LD), t.astype(LD))
    one, flows = np.ones((n, 5)), []
    for _ in range(steps):
        flows.append(fixed[0])
        x, y = step(*fixed, one)[0], step(*fp64, one)[1]
        fl, T = collide_exact(flow, ref[0], im), ref[1].sum(1, keepdims=True)
        tl = ref[1] + omL * (geq(ref[0]) * T - ref[1])
        fixed, fp64, ref = [(streamed(p[0], E2, nx, ny), streamed(p[1], E5, nx, ny))
                            for p in (x, y, (fl, tl))]
    for k in range(2):
        ea, eb = rms(fixed[k] - ref[k]), rms(fp64[k] - ref[k])
        print("tau", tau, ("flow", "temperature")[k], "fixed", ea, "fp64", eb)
        assert ea <= eb / 20
    la = lb = np.ascontiguousarray(rng.standard_normal((n, 5)))
    lr = la.astype(LD)
    for fk in reversed(flows):
        la = streamed(la, E5, nx, ny, -1)
        lb = streamed(lb, E5, nx, ny, -1)
        lr = streamed(lr, E5, nx, ny, -1)
        la, lb = step(fk, one, la)[0][2], step(fk, one, lb)[1][2]
        lr = lr + omL * ((geq(fk.astype(LD)) * lr).sum(1, keepdims=True) - lr)
    ea, eb = rms(la - lr), rms(lb - lr)
    print("tau", tau, "adjoint temperature fixed", ea, "fp64", eb)
    assert ea <= 1.05 * eb


def dissipation_exact(cfg, f, g):
    """Value and source over the weight."""
    F, im, om = f.astype(LD), imult_of(cfg, g), LD(cfg.omega)
    E = E2[:, :2].astype(LD)
    j, rho = F @ E, F.sum(1)
    V = np.einsum("qa,qb,nq->nab", E, E, F) - j[:, :, None] * j[:, None, :]
    V -= np.eye(2).astype(LD) * (rho / 3)[:, None, None]
    tr = V[:, 0, 0] + V[:, 1, 1]
    pe, pj = np.einsum("qa,qb,nab->nq", E, E, V), np.einsum("nab,nb->na", V, j)
    cv = 3 * om * (1 - om / 2)
    jj = (j * j).sum(1)
    return (2 * im * jj + cv / 2 * (V * V).sum((1, 2)),
            4 * im[:, None] * (j @ E.T) + cv * ((pe - tr[:, None] / 3) - 2 * (pj @ E.T)), jj)


@pytest.mark.parametrize("scale", [0.1, 2.0 ** -11])
@pytest.mark.parametrize("size", [0, 0.1, 1, 100])
@pytest.mark.parametrize("amp", [1e-7, 1e-5, 1e-3, 1e-2, 0.08])
@pytest.mark.parametrize("name", ["d2q9_bgk", "d2q9_bgk_rate", "d2q9_mrt"])
def test_reverse_step_with_the_dissipation_source(source_lib, name, amp, size, scale):
    """Adjoints of size times the source, whose units the step takes where it is the
    larger: adjoint and dJ/dgamma within the FP64 operators' error."""
    cfg = model(name).replace(objective=G.OBJ_DISSIPATION, obj_weight=1.0, interp_scale=scale)
    n, rng = 2000, np.random.default_rng(2)
    f, g = states(cfg, n, 5, amp)
    _, src, jj = dissipation_exact(cfg, f, g)
    s = np.abs(src).max(1, keepdims=True).astype(float)
    lo = np.ascontiguousarray(size * s * (1 + 0.3 * rng.standard_normal((n, 9))))
    a, b, da, db = np.zeros((n, 9)), np.zeros((n, 9)), np.zeros(n), np.zeros(n)
    c = cfg.to_c()
    assert source_lib.fixed_source_step(C.byref(c), n, ptr(f), ptr(g), ptr(lo), ptr(a), ptr(da),
                                        ptr(b), ptr(db)) == n
    ref, dim = reverse_exact(cfg, f, imult_of(cfg, g), lo)
    q, gl = LD(cfg.interp_q), g.astype(LD)
    dref = -LD(scale) / 2 * q * (1 + q) / (q + gl) ** 2 * (dim + 2 * jj)
    print(name, amp, size, "fixed", rms(a - ref - src), rms(da - dref), "fp64",
          rms(b - ref - src), rms(db - dref))
    assert rms(a - ref - src) <= 1.05 * rms(b - ref - src)
    assert rms(da - dref) <= 1.05 * rms(db - dref)


@pytest.mark.parametrize("amp", [1e-5, 1e-2, 0.08])
@pytest.mark.parametrize("scale", [0.1, 2.0 ** -11])
def test_dissipation_of_a_flow_without_stresses(lib, scale, amp):  # noqa: F811
    """Where the porosity term is all of it: as exact as FP64 down to the weakest
    porosity that runs in fixed point."""
    cfg = model("d2q9_bgk").replace(objective=G.OBJ_DISSIPATION, obj_weight=1.0,
                                    interp_scale=scale)
    n, rng = 4000, np.random.default_rng(1)
    _, g = states(cfg, n, 41, amp)
    u = amp * rng.uniform(-1, 1, (n, 3)) * [1, 1, 0]
    sc = u @ E2.T
    f = np.ascontiguousarray(W2.astype(float) * (1 + 3 * sc + 4.5 * sc ** 2 -
                                                 1.5 * (u ** 2).sum(1)[:, None]))
    o, s, c = [np.zeros(9 * n) for _ in range(5)], C.c_int(), cfg.to_c()
    assert lib.fixed_dissipation(C.byref(c), n, ptr(f), ptr(g), *[ptr(v) for v in o],
                                 C.byref(s)) == n
    ref = dissipation_exact(cfg, f, g)[0]
    print(scale, amp, "fixed", rms(o[0][:n] - ref), "fp64", rms(o[3][:n] - ref))
    assert rms(o[0][:n] - ref) <= 1.05 * rms(o[3][:n] - ref)


@pytest.mark.parametrize("scale,objective,taken", [
    (0.1, G.OBJ_DISSIPATION, True), (2.0 ** -11, G.OBJ_DISSIPATION, True),
    (0.0, G.OBJ_DISSIPATION, True), (1e-4, G.OBJ_DISSIPATION, False),
    (1e-9, G.OBJ_DISSIPATION, False), (1e-9, G.OBJ_PRESSURE_DROP, True)])
def test_weaker_porosity_keeps_fp64_where_it_shows(lib, scale, objective, taken):  # noqa: F811
    cfg = model("d2q9_bgk").replace(objective=objective, interp_scale=scale)
    f, g = states(cfg, 100, 3, 0.02)
    assert run_forward(lib, cfg, f, g)[0] == (100 if taken else -1)
