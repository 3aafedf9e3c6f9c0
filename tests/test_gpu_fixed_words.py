"""The fixed-point collisions on the GPU (lbm_fixed.cuh) where sums and products
end in whole words of zeros: populations that are multiples of 2^-13 or 2^-29,
dyadic rates, designs and objective weights.  Carries between the two words of
an integer pass through zero there in every sum of the step kernels, which
random states meet once in 2^32 cells.  Each step is compared, from the state
and the adjoint that went into it, with the operators in extended precision:
a lost carry is 2^32 units of 2^-61, some 1e6 times the bounds."""
import numpy as np
import pytest

import lbmgpu as G
import workloads as W
from test_fixed_math_host import E2, E3, E5, LD, W2, W3, W5, collide_exact, reverse_exact

pytestmark = pytest.mark.gpu

# the largest error of a collision (test_fixed_math_host, at the ends of its range)
FORWARD, REVERSE = 2.0 ** -52, 32 * 2.0 ** -57


def config(name, big):
    """big: more cells than two 256-thread blocks on each of 152 SMs (the reverse
    step's three-block variant on D2Q9)."""
    nx, ny, nz = (320, 250, 1) if big else (70, 37, 1)
    if name.startswith("d3q19"):
        nx, ny, nz = (96, 40, 24) if big else (37, 18, 13)
    z = [(5, 6), (8, 8)] if nz > 1 else [(0, 0), (0, 0)]
    inner = dict(interp_scale=0.5, obj_weight=1.0, obj_in=(20, 23, 8, 9) + z[0],
                 obj_out=(16, 16, 12, 12) + z[1])
    if name == "d3q19_mrt":     # rates whose constants are multiples of 2^-6
        return W.duct_3d(nx, ny, nz).replace(
            omega=1.125, mrt=(63 / 64, 63 / 64, 0.75, 0.5625, 1.25, 3.0, -5.5, -0.5), **inner)
    if name == "d3q19_mrt_rates":
        return W.duct_3d(nx, ny, nz).replace(
            omega=1.9, mrt=(1.19, 1.4, 1.2, 1.98, 0.7, 2.5, 4.0, 0.25), **inner)
    if name == "d3q19_bgk":
        return W.duct_3d(nx, ny, nz).replace(collision=G.BGK, omega=1.125, **inner)
    if name == "d2q9_mrt":
        return W.channel_2d(nx, ny, collision=G.MRT).replace(
            omega=1.25, mrt=(1.125, 1.5, 0.75, 0, 0, 0, 0, 0), **inner)
    if name == "thermal":
        # om_T = 1.5 of the fluid, to rounding
        return W.thermal_2d(nx, ny, heat_rate=0.0).replace(
            omega=1.5, diffusivity=1 / 18., objective=G.OBJ_DOMAIN_TEMPERATURE, **inner)
    c = W.channel_2d(nx, ny).replace(omega=1.5 if name == "d2q9_bgk" else 1.9, **inner)
    return c.replace(objective=G.OBJ_DISSIPATION, obj_weight=0.5) if name.endswith("diss") else c


def quantised(cfg, bits, seed):
    """Accepted states of multiples of 2^-bits, a quarter of them symmetric (no
    momentum), some at rest; designs of 0, 1 and values between."""
    rng = np.random.default_rng(seed)
    w = (W3 if cfg.lattice == G.D3Q19 else W2).astype(float)
    n, h = cfg.ncells, (w.size - 1) // 2
    f = w * (1 + 0.15 * rng.uniform(-1, 1, (n, 1))) + 0.012 * rng.uniform(-1, 1, (n, w.size))
    f[::4, h + 1:] = f[::4, 1:h + 1]
    f[2::16] = w
    f = np.maximum(np.round(f * 2.0 ** bits), 2.0 ** (bits - 8)) * 2.0 ** -bits
    if cfg.lattice == G.D2Q9_D2Q5:
        t = W5.astype(float) * rng.uniform(0, 1, (n, 1)) + 0.1 * rng.uniform(-1, 1, (n, 5))
        t[::5] = 0.125
        f = np.hstack([f, np.round(t * 2.0 ** bits) * 2.0 ** -bits])
    g = rng.uniform(0, 1, n)
    g[::3] = 0.0
    g[1::3] = 1.0
    return f, g


def field(cfg, a):
    return a.reshape(cfg.nz, cfg.ny, cfg.nx, -1)


def moved(cfg, a, E, sign):
    """a_q at x + sign e_q (wrapped round, so good away from the faces)."""
    v = field(cfg, a)
    out = [np.roll(v[..., q], [-sign * int(E[q][2]), -sign * int(E[q][1]), -sign * int(E[q][0])],
                   (0, 1, 2)) for q in range(len(E))]
    return np.stack(out, -1).reshape(a.shape)


def inner_cells(cfg, seed, most=3000, near=None):
    """Cells at least two away from every face: all near the marked ones and others."""
    m = np.zeros((cfg.nz, cfg.ny, cfg.nx), dtype=bool)
    z = slice(2, -2) if cfg.nz > 1 else slice(None)
    m[z, 2:-2, 2:-2] = True
    c = np.flatnonzero(m.ravel())
    rng = np.random.default_rng(seed)
    if near is not None:
        c = np.concatenate([c[near[c]], c[~near[c]][:200]])
    return rng.permutation(c)[:most]


def directions(cfg):
    e = (E3 if cfg.lattice == G.D3Q19 else E2).astype(int)
    if cfg.lattice == G.D2Q9_D2Q5:
        return np.vstack([e, np.hstack([E5, np.zeros((5, 1), int)])])
    return e


def imult_of(cfg, g):
    """The design's porosity factor as a double: one minus a quotient, so that its
    rounding (2^-54) would count among the units below."""
    q = cfg.interp_q
    return (0.5 * (cfg.interp_scale * (1.0 - g * (1.0 + q) / (q + g)))).astype(LD)


def om_t(cfg, g):
    q, ck = LD(cfg.ramp_q), LD(cfg.ramp_ck)
    r = (g * (ck * (1 + q) - 1) + 1) / (ck * (1 + q * g))
    return 1 / (3 * LD(cfg.diffusivity) * r + LD(0.5))


def thermal_parts(cfg, f):
    f = f.astype(LD)
    j = (f[:, :9] @ E2.astype(LD))[:, :2]
    return f[:, 9:], 1 + 3 * (j @ E5.T.astype(LD))


def step_exact(cfg, f, g, om=None):
    q = 9 if cfg.lattice == G.D2Q9_D2Q5 else f.shape[1]
    out = collide_exact(cfg, f[:, :q], imult_of(cfg, g))
    if om is None:
        return out
    t, sc = thermal_parts(cfg, f)
    return np.hstack([out, t + om[:, None] * (W5 * t.sum(1, keepdims=True) * sc - t)])


def dissipation_source(cfg, f, g):
    F, im, om = f.astype(LD), imult_of(cfg, g), LD(cfg.omega)
    E = E2[:, :2].astype(LD)
    j, rho = F @ E, F.sum(1)
    V = np.einsum("qa,qb,nq->nab", E, E, F) - j[:, :, None] * j[:, None, :]
    V -= np.eye(2).astype(LD) * (rho / 3)[:, None, None]
    tr = V[:, 0, 0] + V[:, 1, 1]
    pe, pj = np.einsum("qa,qb,nab->nq", E, E, V), np.einsum("nab,nb->na", V, j)
    return LD(cfg.obj_weight) * (4 * im[:, None] * (j @ E.T) + 3 * om * (1 - om / 2) *
                                 ((pe - tr[:, None] / 3) - 2 * (pj @ E.T)))


NAMES = ["d3q19_mrt", "d3q19_mrt_rates", "d3q19_bgk", "d2q9_bgk", "d2q9_bgk_diss",
         "d2q9_bgk_rate_diss", "d2q9_mrt", "d2q9_mrt_diss", "thermal"]


def case(name, big):
    if name == "d2q9_mrt_diss":
        return config("d2q9_mrt", big).replace(objective=G.OBJ_DISSIPATION, obj_weight=0.5)
    return config(name, big)


@pytest.fixture(params=["handle", "batch"])
def opened(request):
    """(name, cfg) -> a handle and the function that takes its forward steps"""
    keep = []

    def open_(name, cfg):
        if request.param == "handle":
            h = G.Handle(cfg)
            keep.append(h)
            return h, h.forward
        b = G.Batch([case(name, False), cfg])
        keep.append(b)
        b[0].set_design(np.ones(b[0].cfg.ncells))
        b[0].init_equilibrium()
        return b[1], b.forward

    yield open_
    for k in keep:
        k.close()


@pytest.mark.parametrize("bits", [13, 29])
@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("name", NAMES)
def test_forward_steps_through_zero_words(opened, name, big, bits):
    cfg = case(name, big)
    f, g = quantised(cfg, bits, 7)
    om = om_t(cfg, g.astype(LD)) if cfg.lattice == G.D2Q9_D2Q5 else None
    h, forward = opened(name, cfg)
    h.set_design(g)
    h.set_populations(f, 400)
    forward(1)
    out = h.populations().reshape(f.shape)
    # the population that arrived at x was collided at x - e_q: move it back
    got = moved(cfg, out, directions(cfg), 1)
    c = inner_cells(cfg, 1)
    ref = step_exact(cfg, f[c], g[c], None if om is None else om[c])
    # om_T of the design is a double made of some eight operations
    bound = FORWARD if om is None else FORWARD + 8 * 2.0 ** -53
    assert np.abs(got[c] - ref).astype(float).max() < bound


def check_reverse(cfg, f, g, lam, out, dg, c):
    """One reverse step: lam the (streamed) adjoint that went in, out what came
    back, dg dJ/dgamma before and after."""
    lo, got, fc, gc = lam[c], moved(cfg, out, directions(cfg), -1)[c], f[c], g[c]
    im = imult_of(cfg, gc)
    ref, dim = reverse_exact(cfg, fc[:, :9 if cfg.lattice == G.D2Q9_D2Q5 else None], im,
                             lo[:, :9 if cfg.lattice == G.D2Q9_D2Q5 else None])
    units = REVERSE * np.abs(lo).max(1, keepdims=True)
    if cfg.objective == G.OBJ_DISSIPATION:
        src = dissipation_source(cfg, fc, gc)
        ref = ref + src
        # its units where the adjoint is smaller (a diagonal adds below 32 of them)
        units = units + 32 * 2.0 ** -61 * abs(cfg.obj_weight)
    if cfg.lattice == G.D2Q9_D2Q5:
        om = om_t(cfg, gc.astype(LD))[:, None]
        t, sc = thermal_parts(cfg, fc)
        l = lo[:, 9:].astype(LD)
        tref = l + om * ((W5 * sc * l).sum(1, keepdims=True) - l)
        ux = om[:, 0] / 2 * t.sum(1) * (l[:, 4] - l[:, 2])
        uy = om[:, 0] / 2 * t.sum(1) * (l[:, 3] - l[:, 1])
        ref = np.hstack([ref + (ux[:, None] * E2[:, 0] + uy[:, None] * E2[:, 1]), tref])
        # the design's om_T is a rounded double: a few 2^-53 of it
        units = units + 8 * 2.0 ** -53 * np.abs(lo).max(1, keepdims=True)
    assert (np.abs(got - ref) <= 2 * 2.0 ** -53 * np.abs(ref) + units).all()
    if dg is not None:
        before, after = [v[c] for v in dg]
        q, gl, s = LD(cfg.interp_q), gc.astype(LD), LD(cfg.interp_scale)
        dimult = -s / 2 * q * (1 + q) / (q + gl) ** 2
        dref = dimult * dim
        # d(imult)/d(gamma) is the difference of two values up to (q + 1) / q times it
        assert (np.abs(after - before - dref) <= 2.0 ** -52 * np.abs(after) +
                64 * 2.0 ** -53 * np.abs(dref) + np.abs(dimult) * units[:, 0]).all()


@pytest.mark.parametrize("bits", [13, 29])
@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("name", NAMES)
def test_reverse_steps_through_zero_words(name, big, bits):
    """Steps from the objective's source alone (zeros and dyadic values), through
    cells at rest and moving, then from what came of them."""
    cfg = case(name, big)
    diss, thermal = cfg.objective == G.OBJ_DISSIPATION, cfg.lattice == G.D2Q9_D2Q5
    with G.Handle(cfg) as h:
        f, g = quantised(cfg, bits, 20)
        h.set_design(g)
        h.set_populations(f, 404)
        h.adjoint_reset()
        lam, s0 = np.zeros(f.shape), np.zeros(cfg.ncells)
        for k in range(4):
            f, _ = quantised(cfg, bits, 20 + k)
            h.set_populations(f, 404 - k)
            h.adjoint_step()
            out, s1 = h.adjoint().reshape(f.shape), h.sensitivity()
            boxes = np.zeros((cfg.nz, cfg.ny, cfg.nx), dtype=bool)
            if not diss:
                for b in (cfg.obj_in, cfg.obj_out):
                    boxes[b[4]:b[5] + 1, b[2]:b[3] + 1, b[0]:b[1] + 1] = True
            near = (lam != 0).any(1) & ~boxes.ravel()
            c = inner_cells(cfg, 2, near=None if diss else near)
            c = c[~boxes.ravel()[c]]
            # dJ/dgamma where no objective or temperature has a share in it
            check_reverse(cfg, f, g, lam, out, None if diss or thermal else (s0, s1), c)
            lam, s0 = out, s1
