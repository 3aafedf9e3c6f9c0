"""The fixed-point collisions of FP64 storage (lbm_fixed.cuh), built for the
host, against the operators in extended precision: over the accepted range
their error is no larger than that of the FP64 operators, they conserve mass
and momentum, and they refuse what lies outside the range.  Runs without a
GPU."""
import ctypes as C
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

import lbmgpu as G
import workloads as W
from test_device_math_host import _cuda_include

HERE = os.path.dirname(os.path.abspath(__file__))
LD = np.longdouble

E2 = np.array([(0, 0, 0), (1, -1, 0), (0, -1, 0), (-1, -1, 0), (-1, 0, 0), (-1, 1, 0), (0, 1, 0),
               (1, 1, 0), (1, 0, 0)])
E3 = np.array([(0, 0, 0), (0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, -1, -1), (0, 1, -1), (-1, 0, -1),
               (1, 0, -1), (-1, -1, 0), (1, -1, 0)])
E3 = np.vstack([E3, -E3[1:]])
W2 = np.array([LD(4) / 9] + [LD(1) / 36, LD(1) / 9] * 4)
W3 = np.array([LD(1) / 3] + 2 * ([LD(1) / 18] * 3 + [LD(1) / 36] * 6))[
    [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18]]


@pytest.fixture(scope="module")
def lib():
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    so = os.path.join(tempfile.mkdtemp(), "libfixedmath.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-ffp-contract=off",
                           "-I" + inc, os.path.join(HERE, "fixed_math_host.cpp"), "-o", so])
    lib = C.CDLL(so)
    dp = C.POINTER(C.c_double)
    lib.fixed_forward.argtypes = [C.POINTER(G.CConfig), C.c_int, dp, dp, dp, dp]
    lib.fixed_reverse.argtypes = [C.POINTER(G.CConfig), C.c_int, dp, dp, dp, dp, dp, dp, dp]
    lib.fixed_thermal.argtypes = [C.c_int] + [dp] * 9
    lib.fixed_dissipation.argtypes = [C.POINTER(G.CConfig), C.c_int] + [dp] * 7 + [C.POINTER(C.c_int)]
    return lib


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def model(name):
    if name == "d3q19_mrt":
        return W.duct_3d(8, 8, 8)
    if name == "d3q19_mrt_rates":
        c = W.duct_3d(8, 8, 8)
        return c.replace(omega=1.9, mrt=(1.19, 1.4, 1.2, 1.98, 0.7, 2.5, 4.0, 0.25))
    if name == "d3q19_bgk":
        return W.duct_3d(8, 8, 8).replace(collision=G.BGK)
    if name == "d2q9_bgk":
        return W.channel_2d(8, 8)
    if name == "d2q9_bgk_rate":
        return W.channel_2d(8, 8, tau=0.52)
    if name == "d2q9_mrt":
        return W.channel_2d(8, 8, collision=G.MRT)
    if name == "d2q9_mrt_rates":
        return W.channel_2d(8, 8, tau=0.51, collision=G.MRT).replace(mrt=(1.1, 1.98, 0.6, 0, 0, 0, 0, 0))
    raise KeyError(name)


def imult_of(cfg, g):
    q, gl = LD(cfg.interp_q), g.astype(LD)
    return LD(cfg.interp_scale) / 2 * q * (1 - gl) / (q + gl)


def collide_exact(cfg, f, im):
    """PBB(base(f)) of the rows of f (n, Q) in extended precision, from the
    moment basis and the equilibrium of each operator."""
    f = f.astype(LD)
    three = cfg.lattice == G.D3Q19
    E, w = (E3, W3) if three else (E2, W2)
    rho, j = f.sum(1), f @ E.astype(LD)
    x, y, z = j.T
    s = x * x + y * y + z * z
    if cfg.collision == G.MRT:
        e = E.astype(int)
        ee = (e * e).sum(1)
        ex, ey, ez = e.T
        if three:
            rows = [1 + 0 * ee, 19 * ee - 30, (21 * ee ** 2 - 53 * ee + 24) // 2, ex,
                    (5 * ee - 9) * ex, ey, (5 * ee - 9) * ey, ez, (5 * ee - 9) * ez,
                    3 * ex ** 2 - ee, (3 * ee - 5) * (3 * ex ** 2 - ee), ey ** 2 - ez ** 2,
                    (3 * ee - 5) * (ey ** 2 - ez ** 2), ex * ey, ey * ez, ex * ez,
                    (ey ** 2 - ez ** 2) * ex, (ez ** 2 - ex ** 2) * ey, (ex ** 2 - ey ** 2) * ez]
            we, wej, wxx = [LD(v) for v in cfg.mrt[5:8]]
            t, u, o = 2 * x * x - y * y - z * z, y * y - z * z, 0 * x
            d = LD(2) / 3
            eq = [rho, -11 * rho + 19 * s, we * rho + wej * s, x, -d * x, y, -d * y, z, -d * z, t,
                  wxx * t, u, wxx * u, x * y, y * z, x * z, o, o, o]
            s1, s2, s4, s10, s16 = [LD(v) for v in cfg.mrt[:5]]
            om = LD(cfg.omega)
            rate = [0, s1, s2, 0, s4, 0, s4, 0, s4, om, s10, om, s10, om, om, om, s16, s16, s16]
        else:
            rows = [1 + 0 * ee, 3 * ee - 4, (9 * ee ** 2 - 21 * ee + 8) // 2, ex, (3 * ee - 5) * ex,
                    ey, (3 * ee - 5) * ey, ex ** 2 - ey ** 2, ex * ey]
            eq = [rho, -2 * rho + 3 * s, rho - 3 * s, x, -x, y, -y, x * x - y * y, x * y]
            s1, s2, s46 = [LD(v) for v in cfg.mrt[:3]]
            rate = [0, s1, s2, 0, s46, 0, s46, LD(cfg.omega), LD(cfg.omega)]
        M = np.array(rows).astype(LD)
        N = (M * M).sum(1)
        r = (f @ M.T - np.array(eq).T) * np.array(rate, dtype=LD)
        f = f - (r / N) @ M
    else:
        sc = j @ E.T.astype(LD)
        om = LD(cfg.omega)
        f = f + om * (w * (rho[:, None] + 3 * sc + sc * sc * 9 / 2 - s[:, None] * 3 / 2) - f)
    im = im[:, None]
    h = (E.shape[0] - 1) // 2
    d = im * (f[:, h + 1:] - f[:, 1:h + 1])
    return np.hstack([f[:, :1], f[:, 1:h + 1] + d, f[:, h + 1:] - d])


def states(cfg, n, seed, amp, rho0=1.0):
    """Equilibria at random density and velocity plus noise, with designs."""
    rng = np.random.default_rng(seed)
    three = cfg.lattice == G.D3Q19
    E, w = (E3, W3) if three else (E2, W2)
    rho = rho0 * (1 + amp * rng.uniform(-1, 1, n))
    u = amp * rng.uniform(-1, 1, (n, 3)) * ([1, 1, 1] if three else [1, 1, 0])
    sc = u @ E.T
    f = w.astype(float) * (rho[:, None] + 3 * sc + 4.5 * sc ** 2 - 1.5 * (u ** 2).sum(1)[:, None])
    f = f * (1 + 0.02 * amp * rng.standard_normal(f.shape))
    g = rng.uniform(0, 1, n)
    g[::5] = 1.0
    g[1::7] = 0.0
    return np.ascontiguousarray(f), np.ascontiguousarray(g)


def run_forward(lib, cfg, f, g):
    c = cfg.to_c()
    a, b = np.empty_like(f), np.empty_like(f)
    taken = lib.fixed_forward(C.byref(c), f.shape[0], ptr(f), ptr(g), ptr(a), ptr(b))
    return taken, a, b


MODELS = ["d3q19_mrt", "d3q19_mrt_rates", "d2q9_bgk", "d2q9_bgk_rate", "d2q9_mrt", "d2q9_mrt_rates",
          "d3q19_bgk"]


@pytest.mark.parametrize("rho0,amp", [(1.0, 1e-6), (1.0, 0.01), (1.0, 0.08), (0.6, 0.08), (1.8, 0.08)])
@pytest.mark.parametrize("name", MODELS)
def test_fixed_forward_is_at_least_as_exact_as_fp64(lib, name, rho0, amp):
    cfg = model(name)
    n = 4000
    f, g = states(cfg, n, 11, amp, rho0)
    taken, a, b = run_forward(lib, cfg, f, g)
    assert taken == n
    ref = collide_exact(cfg, f, imult_of(cfg, g))
    # per direction, over the cells: within the FP64 operator's own error
    # (1.05: both are dominated by the same final rounding where it is small)
    ea = np.sqrt((((a - ref) ** 2).mean(0))).astype(float)
    eb = np.sqrt((((b - ref) ** 2).mean(0))).astype(float)
    print(name, amp, "rms error per direction: fixed", ea.max(), "fp64", eb.max(), "ratio",
          (ea / eb).max())
    assert (ea <= 1.05 * eb).all()
    # mass of the cells: conserved to the rounding of the results, without bias
    dm = (a.astype(LD).sum(1) - f.astype(LD).sum(1)).astype(float)
    assert np.abs(dm).max() < 2.0 ** -52 * max(1.0, rho0)
    assert abs(dm.mean()) < 2.0 ** -57 * max(1.0, rho0)
    # and the momentum of the cells without porosity: the mean error of 800
    # cells is rounding (2^-55 a cell), not a bias
    E = (E3 if cfg.lattice == G.D3Q19 else E2).astype(LD)
    dj = ((a.astype(LD) - f.astype(LD)) @ E)[g == 1.0].astype(float)
    assert np.abs(dj.mean(0)).max() < 2.0 ** -58


def corner_states(cfg, seed, n=3000):
    """States whose populations sit at the ends of the accepted range: each at
    its upper or lower limit at a density of 0.3 to 2.2, along random signs and
    along the signs of every moment row, where the intermediates are largest;
    the rest population completes the density."""
    rng = np.random.default_rng(seed)
    three = cfg.lattice == G.D3Q19
    w = (W3 if three else W2).astype(float)
    E = (E3 if three else E2).astype(int)
    rho = rng.uniform(0.3, 2.2, (n, 1))
    d = 2.0 ** -4 * (1 - 1e-6)
    hi = np.minimum(w * rho + d, 0.5 - 2.0 ** -53)
    lo = np.maximum(w * rho - d, 2.0 ** -9)
    s = rng.integers(0, 2, (n, w.size)).astype(float)
    ee = (E * E).sum(1)
    rows = [ee == 0, ee == 1, ee == 2] + [E[:, a] * E[:, b] > 0 for a in range(3) for b in range(3)]
    rows += [E[:, a] > 0 for a in range(3)] + [E[:, a] ** 2 > E[:, b] ** 2 for a, b in
                                              ((0, 1), (1, 2), (2, 0), (1, 0))]
    for k, r in enumerate(rows):
        s[2 * k], s[2 * k + 1] = r, ~r
    f = lo + s * (hi - lo)
    f[:, 0] = (w[0] * rho + d * (2 * s[:, :1] - 1))[:, 0]
    # pull the others towards their share until the density is right, where it can be
    for _ in range(60):
        r = f.sum(1, keepdims=True)
        off = (r - rho) / (w.size - 1)
        f[:, 1:] = np.clip(f[:, 1:] - off, lo[:, 1:], hi[:, 1:])
    keep = (np.abs(f - w * f.sum(1, keepdims=True)) < d).all(1) & (f[:, 0] < 1) & (f[:, 0] > 2.0 ** -8)
    f = f[keep]
    assert f.shape[0] > 500
    g = rng.uniform(0, 1, f.shape[0])
    g[:50] = 0.0
    return np.ascontiguousarray(f), np.ascontiguousarray(g)


@pytest.mark.parametrize("name", MODELS)
def test_fixed_forward_at_the_ends_of_its_range(lib, name):
    cfg = model(name)
    f, g = corner_states(cfg, 5)
    taken, a, _ = run_forward(lib, cfg, f, g)
    assert taken == f.shape[0]
    # results below 2: half a unit in the last place (2^-53) and the products'
    # few units of 2^-61, times the largest back-map weight (15 units)
    err = np.abs(a - collide_exact(cfg, f, imult_of(cfg, g))).astype(float).max()
    print(name, "largest error", err)
    assert err < 2.0 ** -52


@pytest.mark.parametrize("name", MODELS)
def test_fixed_forward_refuses_what_lies_outside(lib, name):
    """One population of an accepted cell moved past a limit (or the density past
    2.2): the FP64 operator takes the cell, with the same result bit for bit."""
    cfg = model(name)
    w = (W3 if cfg.lattice == G.D3Q19 else W2).astype(float)
    q = w.size
    bad = [-1e-300, 0.0, -0.05, 2.0 ** -9 * (1 - 1e-15), 0.75, 1.0, 3.0, 4.03, 8.2, 1e10, 1e300, np.inf,
           np.nan, 5e-324]
    # an excess x takes the population past its share of the density it adds to
    cells = [(i, v) for i in range(q) for v in bad + [w[i] + 2.0 ** -4 / (1 - w[i]) * (1 + 1e-6),
                                                     w[i] - 2.0 ** -4 / (1 - w[i]) * (1 + 1e-6)]]
    f = np.tile(w, (len(cells), 1))
    for k, (i, v) in enumerate(cells):
        f[k, i] = v
    f = np.vstack([f, w[None] * 2.4 / (1 if q == 9 else 0.75), w[None] * 0.02])
    cells += [None, None]
    g = np.full(len(cells), 0.5)
    taken, a, b = run_forward(lib, cfg, f, g)
    assert taken == 0
    assert np.array_equal(a, b, equal_nan=True)


def reverse_exact(cfg, f, im, lo):
    """Transposed collision of lo and its derivative by imult: the operator is
    quadratic in f and linear in imult, so unit central differences are exact."""
    f, lo = f.astype(LD), lo.astype(LD)
    out = np.empty_like(f)
    for q in range(f.shape[1]):
        e = np.zeros(f.shape[1], dtype=LD)
        e[q] = LD(1) / 4
        d = (collide_exact(cfg, f + e, im) - collide_exact(cfg, f - e, im)) * 2
        out[:, q] = (d * lo).sum(1)
    d = collide_exact(cfg, f, im + 1) - collide_exact(cfg, f, im)
    return out, (d * lo).sum(1)


def run_reverse(lib, cfg, f, g, lo):
    c = cfg.to_c()
    n = f.shape[0]
    a, b = np.empty_like(f), np.empty_like(f)
    da, db = np.empty(n), np.empty(n)
    taken = lib.fixed_reverse(C.byref(c), n, ptr(f), ptr(g), ptr(lo), ptr(a), ptr(da), ptr(b), ptr(db))
    return taken, a, da, b, db


def adjoints(cfg, n, kind, seed=3):
    """Adjoints as the reverse sweep has them: a common value with small
    differences (kind "smooth"), independent values ("rough"), or values of
    very different sizes within a cell ("spread")."""
    rng = np.random.default_rng(seed)
    q = cfg.npop
    scale = 10.0 ** rng.uniform(-12, 2, (n, 1))
    r = rng.standard_normal((n, q))
    if kind == "smooth":
        r = 1 + 0.01 * r
    if kind == "spread":
        r = r * 10.0 ** rng.uniform(-6, 0, (n, q))
    return np.ascontiguousarray(scale * r)


@pytest.mark.parametrize("kind", ["smooth", "rough", "spread"])
@pytest.mark.parametrize("name", MODELS)
def test_fixed_reverse_is_at_least_as_exact_as_fp64(lib, name, kind):
    cfg = model(name)
    n = 3000
    f, g = states(cfg, n, 21, 0.06)
    lo = adjoints(cfg, n, kind)
    taken, a, da, b, db = run_reverse(lib, cfg, f, g, lo)
    assert taken == n
    ref, dref = reverse_exact(cfg, f, imult_of(cfg, g), lo)
    size = np.abs(lo).max(1, keepdims=True)
    ea = np.sqrt((((a - ref) / size) ** 2).mean()).astype(float)
    eb = np.sqrt((((b - ref) / size) ** 2).mean()).astype(float)
    ga = np.sqrt((((da - dref) / size[:, 0]) ** 2).mean()).astype(float)
    gb = np.sqrt((((db - dref) / size[:, 0]) ** 2).mean()).astype(float)
    print(name, kind, "rms error by the cell's largest: fixed", ea, "fp64", eb, "ratio", ea / eb,
          " by imult: fixed", ga, "fp64", gb, "ratio", ga / gb)
    assert ea <= 1.05 * eb
    assert ga <= 1.05 * gb
    # along the common value, which the transposed collision keeps, no bias
    # beyond a unit of the reduced integers (2^-57 of the largest)
    if kind == "smooth":
        assert abs(((a - ref) / size).mean()) < 2.0 ** -57


@pytest.mark.parametrize("name", MODELS)
def test_fixed_reverse_at_the_ends_of_its_range(lib, name):
    """Extreme states with adjoints whose magnitudes are all the cell's
    largest, along random signs and along the signs of the moment rows."""
    cfg = model(name)
    f, g = corner_states(cfg, 6)
    s = corner_states(cfg, 7)[0]
    s = s > (W3 if cfg.lattice == G.D3Q19 else W2).astype(float) * s.sum(1, keepdims=True)
    lo = np.ascontiguousarray((2.0 * np.resize(s, f.shape) - 1) * (2 - 1e-15))
    taken, a, da, _, _ = run_reverse(lib, cfg, f, g, lo)
    assert taken == f.shape[0]
    ref, dref = reverse_exact(cfg, f, imult_of(cfg, g), lo)
    # the result's own rounding and at most 32 units of 2^-57 of the largest
    # (2): a result adds up some 16 products, each within two units
    assert (np.abs(a - ref) <= 2.0 ** -53 * np.abs(ref) + 32 * 2.0 ** -56).all()
    assert (np.abs(da - dref) <= 2.0 ** -53 * np.abs(dref) + 32 * 2.0 ** -56).all()


@pytest.mark.parametrize("name", MODELS)
def test_fixed_reverse_zeros_and_refusals(lib, name):
    cfg = model(name)
    q = cfg.npop
    f, g = states(cfg, 6, 2, 0.05)
    lo = np.zeros((6, q))
    lo[1] = -0.0
    lo[2, 3] = np.nan
    lo[3, 4] = np.inf
    lo[4] = 1e-250
    lo[5] = 1e30
    taken, a, da, b, db = run_reverse(lib, cfg, f, g, lo)
    assert taken == 2
    assert np.array_equal(a[:2], np.zeros((2, q))) and np.array_equal(da[:2], np.zeros(2))
    assert np.array_equal(a[2:], b[2:], equal_nan=True)
    assert np.array_equal(da[2:], db[2:], equal_nan=True)


E5 = np.array([(0, 0), (0, -1), (-1, 0), (0, 1), (1, 0)])
W5 = np.array([LD(1) / 3] + [LD(1) / 6] * 4)


def relative(a, ref, size):
    return np.sqrt((((a - ref) / size) ** 2).mean()).astype(float)


@pytest.mark.parametrize("spread", [0.01, 1.0])
def test_fixed_thermal_is_at_least_as_exact_as_fp64(lib, spread):
    """Collision of the temperature lattice and its transpose at temperatures and
    adjoints of any size (1e-30 to 1e6), near and far from equilibrium."""
    n = 4000
    rng = np.random.default_rng(8)
    f, _ = states(model("d2q9_bgk"), n, 31, 0.08)
    size = 10.0 ** rng.uniform(-30, 6, (n, 1))
    t = np.ascontiguousarray(size * W5.astype(float) * (1 + spread * rng.standard_normal((n, 5))))
    l = np.ascontiguousarray(size[::-1] * (1 + spread * rng.standard_normal((n, 5))))
    t[0], l[1] = 0.0, 0.0
    om = rng.uniform(0.05, 1.98, n)
    out = [np.zeros((n, 5)) for _ in range(4)]
    misc = np.zeros((n, 3))
    assert lib.fixed_thermal(n, ptr(f), ptr(t), ptr(l), ptr(om), *[ptr(v) for v in out], ptr(misc)) == n
    j = (f.astype(LD) @ E2.astype(LD))[:, :2]
    sc = 1 + 3 * (j @ E5.T.astype(LD))
    tl, ll, ol = t.astype(LD), l.astype(LD), om.astype(LD)[:, None]
    ref = tl + ol * (W5 * tl.sum(1, keepdims=True) * sc - tl)
    lref = ll + ol * ((W5 * sc * ll).sum(1, keepdims=True) - ll)
    st = np.maximum(np.abs(t).max(1, keepdims=True), 1e-300)
    sl = np.maximum(np.abs(l).max(1, keepdims=True), 1e-300)
    for a, b, r, s in ((out[0], out[1], ref, st), (out[2], out[3], lref, sl)):
        ea, eb = relative(a, r, s), relative(b, r, s)
        print("thermal", spread, "fixed", ea, "fp64", eb, "ratio", ea / eb)
        assert ea <= 1.05 * eb
    assert not out[0][0].any() and not out[2][1].any()
    keep = np.arange(n) != 1
    for k, v in enumerate((ll[:, 4] - ll[:, 2], ll[:, 3] - ll[:, 1], 2 * ll[:, 0] + ll[:, 1:].sum(1))):
        assert (np.abs(misc[:, k] - v)[keep] <= 2.0 ** -53 * np.abs(v)[keep] + 8 * 2.0 ** -58 * sl[keep, 0]).all()


@pytest.mark.parametrize("weight", [1.0, 5e-4, -3.0])
@pytest.mark.parametrize("amp", [1e-5, 0.01, 0.08])
def test_fixed_dissipation_is_at_least_as_exact_as_fp64(lib, amp, weight):
    """Value, source (added to adjoints of sizes from 2^-40 to 2^20, whose units
    take it or do not) and derivative by imult."""
    cfg = model("d2q9_bgk").replace(obj_weight=weight)
    n = 6100
    f, g = states(cfg, n, 41, amp)
    c = cfg.to_c()
    val, val64, dim = np.zeros(n), np.zeros(n), np.zeros(n)
    src, src64 = np.zeros((n, 9)), np.zeros((n, 9))
    scaled = C.c_int()
    assert lib.fixed_dissipation(C.byref(c), n, ptr(f), ptr(g), ptr(val), ptr(src), ptr(dim),
                                 ptr(val64), ptr(src64), C.byref(scaled)) == n
    assert n // 4 < scaled.value < n
    F, im, om = f.astype(LD), imult_of(cfg, g), LD(cfg.omega)
    E = E2[:, :2].astype(LD)
    j, rho = F @ E, F.sum(1)
    V = np.einsum("qa,qb,nq->nab", E, E, F) - j[:, :, None] * j[:, None, :]
    V -= np.eye(2).astype(LD) * (rho / 3)[:, None, None]
    cv = LD(3) / 2 * om * (1 - om / 2)
    ref = 2 * im * (j * j).sum(1) + cv * (V * V).sum((1, 2))
    tr = V[:, 0, 0] + V[:, 1, 1]
    pe = np.einsum("qa,qb,nab->nq", E, E, V)
    pj = np.einsum("nab,nb->na", V, j)
    sref = 4 * im[:, None] * (j @ E.T) + 2 * cv * ((pe - tr[:, None] / 3) - 2 * (pj @ E.T))
    w = LD(weight)
    # the source's error where the adjoint it joins is no larger than the weight
    # (else it is the adjoint's own rounding that counts)
    small = (np.arange(n) % 61 - 40) <= np.log2(abs(weight))
    ea, eb = relative(val, w * ref, w), relative(val64, w * ref, w)
    sa, sb = relative(src[small], (w * sref)[small], w), relative(src64[small], (w * sref)[small], w)
    print("dissipation", amp, "value: fixed", ea, "fp64", eb, "source: fixed", sa, "fp64", sb)
    assert ea <= 1.05 * eb and sa <= 1.05 * sb
    size = 1.3 * 2.0 ** (np.arange(n) % 61 - 40)
    # a diagonal population adds two components of g (four-fold products of
    # V j, each of four products) and an even part: below 32 units in all
    assert (np.abs(src - w * sref).astype(float) <=
            (32 * 2.0 ** -61 * abs(weight) + 8 * 2.0 ** -57 * size)[:, None] +
            2.0 ** -53 * np.abs(w * sref).astype(float)).all()
    # three roundings of 2 j^2 <= 4 (1.2 amp)^2, and j itself within 2^-61
    assert np.abs(dim - 2 * (j * j).sum(1)).max() < 3 * 2.0 ** -53 * 6 * amp * amp + 2.0 ** -58 * amp
