"""The work that users of this library have it do, as cases to measure: whole
calls of the public entry points (lbmgpu.Handle, Batch, TopOpt) on set-ups of
workloads.py, with seeded designs, over the sizes, lattices, storage types and
drivers that the library's own workloads, tests and benchmark use.

listed() names the cases, draw(rng) gives more of the same ranges, prepare()
makes what a program has in hand before the call, run() is one call, work()
what it cannot do without, and exact() the result in 64 bits from a plain
torch restatement of the same model (forward steps and automatic
differentiation).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "lbm-topopt_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import lbmgpu as G  # noqa: E402
import workloads as W  # noqa: E402

STORES = {64: G.STORE_FP64, 32: G.STORE_FP32, 16: G.STORE_FP16}
LATTICES = {"channel": G.D2Q9, "pump": G.D2Q9, "thermal": G.D2Q9_D2Q5,
            "regenerator": G.D2Q9_D2Q5, "duct": G.D3Q19}
NPOP = {G.D2Q9: 9, G.D2Q9_D2Q5: 14, G.D3Q19: 19}
# floating-point operations of one cell's forward and reverse step, counted
# once from the formulas of the collision operators (a rough figure: the work
# of a step is its bytes)
FLOPS = {G.D2Q9: (150, 300), G.D2Q9_D2Q5: (210, 430), G.D3Q19: (400, 800)}


# ---------------------------------------------------------------------------
# The cases.

def listed():
    return [
        # the smallest calls: a driver in the reference's style that advances a
        # small channel step by step, one call per step (latency and launches)
        dict(name="channel_stepwise_fp64_64x48", kind="stepwise", model="channel", bits=64,
             collision="bgk", nx=64, ny=48, nz=1, steps=8, objective="pressure"),
        # the library's smallest workload, whole: 2000 steps of a 128x64 channel
        # in FP64 (the default and the reference's type), 64 checkpoints
        dict(name="channel_gradient_fp64_128x64", kind="gradient", model="channel", bits=64,
             collision="bgk", nx=128, ny=64, nz=1, steps=2000, snaps=64, objective="pressure"),
        # the robust pump's problem: MRT, oscillating tabulated inlet, odd size
        dict(name="pump_gradient_fp64_201x201", kind="gradient", model="pump", bits=64,
             collision="mrt", nx=201, ny=201, nz=1, steps=600, snaps=20, objective="through"),
        # the unsteady channel with the dissipation objective, in the production
        # storage type and in FP64 (its states stay in the GPU's L2)
        dict(name="channel_gradient_fp32_1024x512", kind="gradient", model="channel", bits=32,
             collision="bgk", nx=1024, ny=512, nz=1, steps=1000, snaps=64,
             objective="dissipation"),
        dict(name="channel_gradient_fp64_1024x512", kind="gradient", model="channel", bits=64,
             collision="bgk", nx=1024, ny=512, nz=1, steps=200, snaps=32,
             objective="dissipation"),
        # heated obstacle: flow and temperature lattices, heat flux
        dict(name="thermal_gradient_fp32_512x256", kind="gradient", model="thermal", bits=32,
             collision="bgk", nx=512, ny=256, nz=1, steps=1000, snaps=64, objective="heat"),
        # the regenerator's driver: steady phase, ramp, unsteady objective; ragged size
        dict(name="regenerator_steady_fp64_255x97", kind="steady", model="regenerator", bits=64,
             collision="bgk", nx=255, ny=97, nz=1, steps=200, snaps=24, max_steady=400,
             check=100, objective="efficiency"),
        # the benchmark's duct (larger than L2): gradient in the production type
        dict(name="duct_gradient_fp32_256x128x128", kind="gradient", model="duct", bits=32,
             collision="mrt", nx=256, ny=128, nz=128, steps=200, snaps=32, objective="pressure"),
        # the same duct at an eighth of the size in FP64
        dict(name="duct_gradient_fp64_128x64x64", kind="gradient", model="duct", bits=64,
             collision="mrt", nx=128, ny=64, nz=64, steps=100, snaps=16, objective="pressure"),
        # a forward simulation with half-width storage and a look at its fields,
        # ragged, with the objective of every step
        dict(name="duct_forward_fp16_250x121x115", kind="forward", model="duct", bits=16,
             collision="mrt", nx=250, ny=121, nz=115, steps=200, objective="pressure"),
        # an ensemble: eight uneven channels stepped together, graph replay
        dict(name="batch_gradient_fp32_8_channels", kind="batch", model="channel", bits=32,
             collision="bgk", nx=1024, ny=512, nz=1, steps=300, snaps=32, n=8,
             objective="pressure"),
        # the design update of the robust iteration: double projection of three
        # realisations, chain rule, volume constraint and one MMA step
        dict(name="robust_update_1024x512", kind="design", model="channel", bits=64,
             nx=1024, ny=512, nz=1, radius=8, radius2=4, nreal=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stepwise", "gradient", "gradient", "gradient", "gradient", "forward",
                       "forward", "steady", "batch", "design"])
    bits = rng.choice([64, 64, 32, 32, 16])
    if kind == "stepwise":
        return dict(kind=kind, model="channel", bits=rng.choice([64, 64, 32]),
                    collision=rng.choice(["bgk", "mrt"]), nx=_log_int(rng, 24, 240),
                    ny=_log_int(rng, 16, 120), nz=1, steps=rng.randint(4, 24),
                    objective=rng.choice(["pressure", "dissipation"]))
    if kind == "steady":
        nx, ny = _log_int(rng, 96, 512), _log_int(rng, 40, 200)
        return dict(kind=kind, model="regenerator", bits=64, collision="bgk", nx=nx, ny=ny, nz=1,
                    steps=rng.randint(60, 240), snaps=rng.randint(8, 40),
                    max_steady=rng.choice([200, 300, 400]), check=rng.choice([50, 100]),
                    objective=rng.choice(["efficiency", "temperature"]))
    if kind == "batch":
        return dict(kind=kind, model="channel", bits=rng.choice([64, 32, 32]), collision="bgk",
                    nx=_log_int(rng, 128, 1024), ny=_log_int(rng, 64, 512), nz=1,
                    steps=rng.randint(40, 160), snaps=rng.randint(8, 32), n=rng.randint(2, 8),
                    objective=rng.choice(["pressure", "dissipation"]))
    if kind == "design":
        nreal = rng.choice([1, 2, 3])
        if rng.random() < 0.3:
            return dict(kind=kind, model="duct", bits=64, nx=_log_int(rng, 32, 160),
                        ny=_log_int(rng, 24, 80), nz=_log_int(rng, 16, 80),
                        radius=rng.randint(2, 5), radius2=rng.choice([0, 2]), nreal=nreal)
        return dict(kind=kind, model="channel", bits=64, nx=_log_int(rng, 96, 1400),
                    ny=_log_int(rng, 48, 700), nz=1, radius=rng.randint(2, 12),
                    radius2=rng.choice([0, 2, 4]), nreal=nreal)
    model = rng.choice(["channel", "channel", "pump", "thermal", "duct", "duct"])
    collision, objective, nz = "bgk", "pressure", 1
    if model == "duct":
        nx, ny, nz = _log_int(rng, 32, 256), _log_int(rng, 16, 128), _log_int(rng, 16, 128)
        collision = rng.choice(["mrt", "mrt", "mrt", "bgk"])
    elif model == "pump":
        nx = ny = 3 * _log_int(rng, 20, 170)
        collision, objective = rng.choice(["mrt", "mrt", "bgk"]), "through"
    elif model == "thermal":
        nx, ny, objective = _log_int(rng, 64, 768), _log_int(rng, 32, 384), "heat"
    else:
        nx, ny = _log_int(rng, 64, 1600), _log_int(rng, 32, 800)
        collision = rng.choice(["bgk", "bgk", "mrt"])
        objective = rng.choice(["pressure", "dissipation"])
    # as many steps as 40,000 MB of population traffic allow, 30 to 1500
    npop = NPOP[LATTICES[model]]
    step_mb = nx * ny * nz * npop * (bits / 8.0) * (2 if kind == "forward" else 7) / 1e6
    if bits == 64:
        step_mb *= 4
    most = int(max(30, min(1500, 40000.0 / step_mb)))
    steps = rng.randint(30, most)
    case = dict(kind=kind, model=model, bits=bits, collision=collision, nx=nx, ny=ny, nz=nz,
                steps=steps, objective=objective)
    if kind == "gradient":
        case["snaps"] = rng.randint(8, max(9, min(64, steps)))
    return case


# ---------------------------------------------------------------------------
# Set-ups.

def _config(case, nx=None, ny=None):
    nx, ny, nz = nx or case["nx"], ny or case["ny"], case["nz"]
    storage = STORES[case["bits"]]
    collision = G.MRT if case.get("collision") == "mrt" else G.BGK
    steps = case.get("steps", 1)
    if case["model"] == "duct":
        return W.duct_3d(nx, ny, nz, storage=storage, nsteps=steps).replace(collision=collision)
    if case["model"] == "thermal":
        # the heat carried through the middle half of the channel: short runs
        # bring no heat to the outlet
        return W.thermal_2d(nx, ny, storage=storage, period=200.0, nsteps=steps).replace(
            obj_out=(nx // 4, 3 * nx // 4, 1, ny - 2, 0, 0))
    if case["model"] == "pump":
        return W.pump_2d(nx, collision=collision, storage=storage, nsteps=steps)
    if case["model"] == "regenerator":
        obj = (G.OBJ_REGENERATOR_EFFICIENCY if case["objective"] == "efficiency"
               else G.OBJ_DOMAIN_TEMPERATURE)
        return W.regenerator_2d(nx, ny, ramp=60.0, storage=storage, n_unsteady=steps,
                                objective=obj)
    if case["objective"] == "dissipation":
        return W.channel_2d(nx, ny, amp=0.2, period=200.0, storage=storage, collision=collision,
                            objective=G.OBJ_DISSIPATION, nsteps=steps)
    return W.channel_2d(nx, ny, storage=storage, collision=collision, nsteps=steps)


def _blur(a):
    """Mean over the 3x3 (2D) or 3x3x3 neighbourhood with edge replication."""
    d = a.dim()
    pool = torch.nn.functional.avg_pool2d if d == 2 else torch.nn.functional.avg_pool3d
    v = torch.nn.functional.pad(a[None, None], (1, 1) * d, mode="replicate")
    return pool(v, 3, 1)[0, 0]


def _design(model, nx, ny, nz, seed, k=0):
    """A design as an optimisation meets it: noise blurred once (2D channels and
    pumps), thresholded noise with soft interfaces (ducts), a heated disc
    (thermal) or plates (regenerator)."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 7919 * k + 1)
    if model == "thermal":
        r = torch.rand(3, generator=gen, device="cuda", dtype=torch.float64).tolist()
        y, x = torch.meshgrid(torch.arange(ny, device="cuda", dtype=torch.float64),
                              torch.arange(nx, device="cuda", dtype=torch.float64), indexing="ij")
        d = torch.sqrt((x - nx * (0.3 + 0.2 * r[0])) ** 2 + (y - ny * (0.35 + 0.3 * r[1])) ** 2)
        g = (d - ny * (0.12 + 0.06 * r[2])).clamp(0.0, 1.0)
    elif model == "regenerator":
        r = torch.rand(6, generator=gen, device="cuda", dtype=torch.float64).tolist()
        g = torch.ones(ny, nx, device="cuda", dtype=torch.float64)
        for j in range(3):
            x0, w = int(nx * (0.3 + 0.15 * j + 0.05 * r[j])), max(3, int(nx * (0.04 + 0.02 * r[3 + j])))
            y0, y1 = (1, int(ny * 0.45)) if j % 2 == 0 else (int(ny * 0.55), ny - 2)
            g[y0:y1, x0:x0 + w] = 0.0
        g = _blur(g)
    elif nz > 1:
        g = torch.rand(nz, ny, nx, generator=gen, device="cuda", dtype=torch.float64)
        g = _blur((_blur(_blur(g)) >= 0.5).double())
    else:
        g = _blur(torch.rand(ny, nx, generator=gen, device="cuda", dtype=torch.float64))
    return g.clamp(0.0, 1.0).reshape(-1).cpu().numpy()


def _batch_grids(case):
    """Uneven lattices of a batch: the first three of full size, the others
    between a quarter and three quarters of it, as in the eight-channel set."""
    share = [1.0, 1.0, 1.0, 0.25, 0.375, 0.5, 0.625, 0.75][: case["n"]]
    return [(max(16, int(case["nx"] * s)), max(12, int(case["ny"] * s))) for s in share]


def _design_update(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cl = max(2, nx // 16)
    box = (cl, nx - 1 - cl, 1, ny - 2, 1 if nz > 1 else 0, nz - 2 if nz > 1 else 0)
    stages = [(case["radius"], True, 2.0, 0.5)]
    if case["radius2"]:
        stages.append((case["radius2"], True, 8.0, 0.5))
    etas = [0.5] if case["nreal"] == 1 else [0.3, 0.5, 0.7][: case["nreal"]]
    n = (box[1] - box[0] + 1) * (box[3] - box[2] + 1) * (box[5] - box[4] + 1)
    return box, stages, etas, n


def _design_inputs(case, seed):
    """Design variables on the box and per realisation (J, dJ/dgamma): smooth
    positive and negative sensitivities of the size the channel's have."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    box, _, etas, n = _design_update(case)
    x = _design("noise", nx, ny, nz if nz > 1 else 1, seed).reshape(nz, ny, nx)
    x = x[box[4]:box[5] + 1, box[2]:box[3] + 1, box[0]:box[1] + 1].reshape(-1).copy()
    assert x.size == n
    sens = []
    for r in range(len(etas)):
        gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 31 * r + 5)
        v = torch.randn((ny, nx) if nz == 1 else (nz, ny, nx), generator=gen, device="cuda",
                        dtype=torch.float64)
        v = 1.0e-6 * (_blur(v) - 0.2)
        sens.append((0.05 + 0.01 * r, v.reshape(-1).cpu().numpy()))
    return x, sens


def prepare(case, seed):
    kind = case["kind"]
    if kind == "design":
        box, stages, etas, n = _design_update(case)
        x, sens = _design_inputs(case, seed)
        t = G.TopOpt(case["nx"], case["ny"], case["nz"], box, stages, nreal=len(etas),
                     real_eta=etas if len(etas) > 1 else None, volume_type=G.VOLUME_FLUID,
                     volume=0.6, move_limit=0.1, x0=x)
        return dict(case=case, topopt=t, x=x, sens=sens)
    if kind == "batch":
        grids = _batch_grids(case)
        b = G.Batch([_config(case, nx, ny) for nx, ny in grids])
        gammas = [_design(case["model"], nx, ny, 1, seed, k) for k, (nx, ny) in enumerate(grids)]
        return dict(case=case, batch=b, gammas=gammas)
    cfg = _config(case)
    h = G.Handle(cfg)
    if case["model"] == "pump":
        h.set_bc_profile(2, W.pump_inflow_profile(cfg))
    gamma = _design(case["model"], case["nx"], case["ny"], case["nz"], seed)
    h.set_design(gamma)
    h.init_equilibrium()
    return dict(case=case, handle=h, gamma=gamma)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "design":
        # one iteration's design update: the physical fields the solver takes,
        # the chain rule of every realisation, the volume constraint and MMA
        t = state["topopt"]
        t.set_variables(state["x"])
        out = {"gamma": [t.physical(r) for r in range(t.nreal)], "dJdx": []}
        for r, (J, s) in enumerate(state["sens"]):
            t.set_sensitivity_host(r, s, J)
            out["dJdx"].append(t.design_sensitivity(r))
        out["change"], out["constraints"] = t.update()
        out["x"] = t.variables()
        return out
    if kind == "batch":
        b = state["batch"]
        for k, g in enumerate(state["gammas"]):
            b[k].set_design(g)
        J, sens, st = b.gradient(case["steps"], case["snaps"], use_graph=True,
                                 schedule=G.SCHEDULE_STATIC)
        return {"J": J, "dJdgamma": sens, "recomputed": int(st.recomputed_steps)}
    h = state["handle"]
    if kind == "stepwise":
        h.init_equilibrium()
        J = [h.forward(1) for _ in range(case["steps"])]
        return {"J": np.array(J), "populations": h.populations(), "macros": h.macros()}
    if kind == "forward":
        h.init_equilibrium()
        J, js = h.forward(case["steps"], per_step=True)
        return {"J": J, "steps": js, "macros": h.macros(), "populations": h.populations()}
    h.set_design(state["gamma"])
    if kind == "steady":
        J, s, st, n = h.gradient_steady(case["max_steady"], case["check"], 1e-7, case["steps"],
                                        case["snaps"])
        return {"J": J, "dJdgamma": s, "steady": int(n), "recomputed": int(st.recomputed_steps)}
    J, s, st = h.gradient(case["steps"], case["snaps"])
    return {"J": J, "dJdgamma": s, "recomputed": int(st.recomputed_steps)}


def work(case):
    """Bytes and operations of one pass.  A forward step reads and writes every
    population and reads the design; a reverse step reads the state and the
    adjoint, writes the adjoint, and updates dJ/dgamma.  Recomputed steps are
    not counted (with every state kept there are none)."""
    if case["kind"] == "design":
        box, stages, etas, n = _design_update(case)
        cells = case["nx"] * case["ny"] * case["nz"]
        taps = 0.0
        for rad, _, _, _ in stages:
            taps += (math.pi * rad ** 2 if case["nz"] == 1 else 4.0 / 3.0 * math.pi * rad ** 3)
        nreal, m = len(etas), (len(etas) if len(etas) > 1 else 0) + 1
        # the fields of every realisation in and out once, and the MMA
        # variables of a pass over its dual: about 60 passes
        b = 8.0 * (cells * nreal * 2 + n * (2 + nreal) + 60.0 * n * (4 + 2 * m))
        return {"bytes": b, "flops": 2.0 * taps * n * (2 * nreal + 2) + 60.0 * n * (20 + 12 * m)}
    grids = _batch_grids(case) if case["kind"] == "batch" else [(case["nx"], case["ny"])]
    cells = sum(nx * ny for nx, ny in grids) * case["nz"]
    lat = LATTICES[case["model"]]
    q, s = NPOP[lat], case["bits"] // 8
    sa, sg = (8, 8) if case["bits"] == 64 else (4, 4)
    fwd = 2 * q * s + sg
    rev = 2 * q * sa + q * s + sg + 16
    f, r = FLOPS[lat]
    steps = case["steps"]
    if case["kind"] in ("stepwise", "forward"):
        out = 8.0 * cells * (q + 4)
        return {"bytes": float(cells) * steps * fwd + out, "flops": float(cells) * steps * f}
    if case["kind"] == "steady":
        steps += case["max_steady"]
    return {"bytes": float(cells) * steps * (fwd + rev) + 16.0 * cells,
            "flops": float(cells) * steps * (f + r)}


# ---------------------------------------------------------------------------
# The same models in plain torch, in 64 bits.

_E2 = [(0, 0), (1, -1), (0, -1), (-1, -1), (-1, 0), (-1, 1), (0, 1), (1, 1), (1, 0)]
_W2 = [4 / 9] + [1 / 36, 1 / 9] * 4
_E3 = [(0, 0, 0), (0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, -1, -1), (0, 1, -1), (-1, 0, -1),
       (1, 0, -1), (-1, -1, 0), (1, -1, 0)]
_E3 = _E3 + [(-a, -b, -c) for a, b, c in _E3[1:]]
_W3 = ([1 / 3] + [1 / 18] * 3 + [1 / 36] * 6) + ([1 / 18] * 3 + [1 / 36] * 6)
_E5 = [(0, 0), (0, -1), (-1, 0), (0, 1), (1, 0)]
_W5 = [1 / 3] + [1 / 6] * 4


class _Model:
    """One lattice of a Config in torch: populations (Q, nz, ny, nx) in FP64."""

    def __init__(self, cfg, table=None):
        self.c, self.table = cfg, table
        dev = dict(device="cuda", dtype=torch.float64)
        three = cfg.lattice == G.D3Q19
        self.three, self.heat = three, cfg.lattice == G.D2Q9_D2Q5
        self.e = _E3 if three else [(a, b, 0) for a, b in _E2]
        w = _W3 if three else _W2
        self.q, self.half = len(self.e), (len(self.e) - 1) // 2
        self.shape = (cfg.nz if three else 1, cfg.ny, cfg.nx)
        self.E = torch.tensor(self.e, **dev)
        self.w = torch.tensor(w, **dev)
        self.opp = [0] + [i + self.half if i <= self.half else i - self.half
                          for i in range(1, self.q)]
        self.e5 = [(a, b, 0) for a, b in _E5]
        self.opp5 = [0, 3, 4, 1, 2]
        self.inside = {}
        for e in set(self.e) | set(self.e5):
            m = torch.ones(self.shape, device="cuda", dtype=torch.bool)
            for axis, d in ((2, e[0]), (1, e[1]), (0, e[2])):
                if d:   # cells whose upstream neighbour x - e lies outside
                    m.narrow(axis, 0 if d > 0 else self.shape[axis] - 1, 1).fill_(False)
            self.inside[e] = m
        if cfg.collision == G.MRT:
            self._mrt(dev)

    def _mrt(self, dev):
        E = [tuple(int(v) for v in e) for e in self.e]
        rows, eq = [], []
        if self.three:
            for x, y, z in E:
                s = x * x + y * y + z * z
                rows.append([1, 19 * s - 30, (21 * s * s - 53 * s + 24) // 2, x, (5 * s - 9) * x, y,
                             (5 * s - 9) * y, z, (5 * s - 9) * z, 3 * x * x - s,
                             (3 * s - 5) * (3 * x * x - s), y * y - z * z,
                             (3 * s - 5) * (y * y - z * z), x * y, y * z, x * z,
                             (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z])
            s1, s2, s4, s10, s16 = list(self.c.mrt)[:5]
            om = self.c.omega
            rate = [0, s1, s2, 0, s4, 0, s4, 0, s4, om, s10, om, s10, om, om, om, s16, s16, s16]
        else:
            for x, y, _ in E:
                s = x * x + y * y
                rows.append([1, 3 * s - 4, (9 * s * s - 21 * s + 8) // 2, x, (3 * s - 5) * x, y,
                             (3 * s - 5) * y, x * x - y * y, x * y])
            s1, s2, s46 = list(self.c.mrt)[:3]
            rate = [0, s1, s2, 0, s46, 0, s46, self.c.omega, self.c.omega]
        self.M = torch.tensor(rows, **dev).t().contiguous()
        self.back = torch.linalg.inv(self.M) * torch.tensor(rate, **dev)[None, :]

    def macros(self, f):
        rho = f[: self.q].sum(0)
        j = torch.einsum("qa,qzyx->azyx", self.E, f[: self.q])
        return rho, j

    def porosity(self, g):
        c = self.c
        return 0.5 * c.interp_scale * (c.interp_q * (1 - g) / (c.interp_q + g))

    def equilibrium(self, rho, j):
        sc = torch.einsum("qa,azyx->qzyx", self.E, j)
        return self.w[:, None, None, None] * (rho + 3 * sc + 4.5 * sc * sc - 1.5 * (j * j).sum(0))

    def start(self):
        rho = torch.ones(self.shape, device="cuda", dtype=torch.float64)
        f = self.equilibrium(rho, torch.zeros(3, *self.shape, device="cuda", dtype=torch.float64))
        return torch.cat([f, torch.zeros(5, *self.shape, device="cuda", dtype=torch.float64)]
                         ) if self.heat else f

    def collide(self, f, g):
        c, q = self.c, self.q
        rho, j = self.macros(f)
        flow = f[:q]
        if c.collision == G.MRT:
            m = torch.einsum("kq,qzyx->kzyx", self.M, flow)
            x, y, z = j
            s = (j * j).sum(0)
            if self.three:
                we, wej, wxx = list(c.mrt)[5:8]
                pxx, pww = 2 * x * x - y * y - z * z, y * y - z * z
                o = torch.zeros_like(rho)
                eq = [rho, -11 * rho + 19 * s, we * rho + wej * s, x, -2 / 3 * x, y, -2 / 3 * y,
                      z, -2 / 3 * z, pxx, wxx * pxx, pww, wxx * pww, x * y, y * z, x * z, o, o, o]
            else:
                eq = [rho, -2 * rho + 3 * s, rho - 3 * s, x, -x, y, -y, x * x - y * y, x * y]
            flow = flow - torch.einsum("qk,kzyx->qzyx", self.back, m - torch.stack(eq))
        else:
            flow = (1 - c.omega) * flow + c.omega * self.equilibrium(rho, j)
        a, h = self.porosity(g), self.half
        d = a * (flow[h + 1:] - flow[1:h + 1])
        flow = torch.cat([flow[:1], flow[1:h + 1] + d, flow[h + 1:] - d])
        if not self.heat:
            return flow
        t = f[q:]
        T = t.sum(0)
        ramp = (g * (c.ramp_ck * (1 + c.ramp_q) - 1) + 1) / (c.ramp_ck * (1 + c.ramp_q * g))
        om = 1 / (3 * c.diffusivity * ramp + 0.5)
        hs = (1 - g) * c.heat_rate * (c.heat_T - T)
        out = [(1 - om) * t[i] + om * _W5[i] * T * (1 + 3 * (e[0] * j[0] + e[1] * j[1]))
               + _W5[i] * hs for i, e in enumerate(self.e5)]
        return torch.cat([flow, torch.stack(out)])

    def stream(self, f):
        out = []
        for es, opp, base in ((self.e, self.opp, 0),) + (
                ((self.e5, self.opp5, self.q),) if self.heat else ()):
            for i, e in enumerate(es):
                moved = torch.roll(f[base + i], (e[2], e[1], e[0]), (0, 1, 2))
                out.append(torch.where(self.inside[e], moved, f[base + opp[i]]))
        return torch.stack(out)

    def _law(self, b, t, t0):
        if b.time_law == G.TIME_SINE:
            return b.amp * math.sin(2 * math.pi * t / b.period)
        if b.time_law == G.TIME_RAMP:
            s = -1 if t0 is None else t - t0
            return b.amp + (0 if s <= 0 else 1 if s >= b.period
                            else math.sin(math.pi * s / (2 * b.period)))
        return 1 + b.amp * math.sin(2 * math.pi * t / b.period)

    def _profile(self, b):
        x0, x1, y0, y1, z0, z1 = b.box
        if b.profile == G.PROFILE_TABLE:
            return torch.from_numpy(self.table[0]).cuda()[None, None, :]
        if b.profile != G.PROFILE_PARABOLIC:
            return 1.0
        def para(n, a, b):
            m = (n - 1) / 2
            v = torch.arange(a, b + 1, device="cuda", dtype=torch.float64)
            return (m * m - (v - m) ** 2) / (m * m)
        p = para(self.c.ny, y0, y1)[None, :, None]
        return p * para(self.c.nz, z0, z1)[:, None, None] if self.three else p

    def boundaries(self, f, t, t0):
        f = f.clone()
        for b in self.c.bcs:
            x0, x1, y0, y1, z0, z1 = b.box
            at = (slice(z0, z1 + 1), slice(y0, y1 + 1), slice(x0, x1 + 1))
            k = [f[(i,) + at].clone() for i in range(f.shape[0])]
            v = b.value * self._law(b, t, t0) * self._profile(b)
            new = {}
            if b.kind == G.BC_TEMPERATURE:
                new[13] = v - k[9] - k[10] - k[11] - k[12]
            elif self.three:
                ny = 0.5 * (k[5] + k[11] + k[13] - k[2] - k[4] - k[14])
                nz = 0.5 * (k[10] + k[13] + k[14] - k[1] - k[4] - k[5])
                if b.kind == G.BC_VELOCITY:
                    new = {7: k[16] + v / 6 + nz, 9: k[18] + v / 6 + ny, 12: k[3] + v / 3,
                           15: k[6] + v / 6 - nz, 17: k[8] + v / 6 - ny}
                else:
                    u = (k[0] + k[1] + k[2] + k[4] + k[5] + k[10] + k[11] + k[13] + k[14]
                         + 2 * (k[7] + k[9] + k[12] + k[15] + k[17])) - v
                    new = {3: k[12] - u / 3, 6: k[15] - u / 6 + nz, 8: k[17] - u / 6 + ny,
                           16: k[7] - u / 6 - nz, 18: k[9] - u / 6 - ny}
            elif b.kind == G.BC_VELOCITY and b.face == G.FACE_WEST:
                d = 0.5 * (k[6] - k[2])
                new = {1: k[5] + d + v / 6, 7: k[3] - d + v / 6, 8: k[4] + 2 / 3 * v}
            elif b.kind == G.BC_VELOCITY:   # north, velocity v * dir with dir along y
                u, d = v * b.dir[1], 0.5 * (k[4] - k[8])
                new = {1: k[5] + d - u / 6, 2: k[6] - 2 / 3 * u, 3: k[7] - d - u / 6}
            else:
                d = 0.5 * (k[6] - k[2])
                if b.face == G.FACE_EAST:
                    u = k[0] + k[2] + k[6] + 2 * (k[1] + k[7] + k[8]) - v
                    new = {4: k[8] - 2 / 3 * u, 3: k[7] - u / 6 + d, 5: k[1] - u / 6 - d}
                else:
                    u = v - (k[0] + k[2] + k[6] + 2 * (k[3] + k[4] + k[5]))
                    new = {8: k[4] + 2 / 3 * u, 7: k[3] + u / 6 - d, 1: k[5] + u / 6 + d}
            for i, val in new.items():
                f[(i,) + at] = val
        return f

    def step(self, f, g, t, t0=None):
        """f_{t+1} from f_t (post-boundary states)."""
        return self.boundaries(self.stream(self.collide(f, g)), t + 1, t0)

    def objective(self, f, g):
        c = self.c
        rho, j = self.macros(f)

        def box(b, v):
            return v[b[4]:b[5] + 1, b[2]:b[3] + 1, b[0]:b[1] + 1]
        o = c.objective
        if o == G.OBJ_PRESSURE_DROP:
            v = box(c.obj_in, rho).mean() - box(c.obj_out, rho).mean()
        elif o == G.OBJ_THROUGH_FLOW:
            v = -box(c.obj_in, j[0]).mean() - box(c.obj_out, j[0]).mean()
        elif o == G.OBJ_DISSIPATION:
            nu = (1 / c.omega - 0.5) / 3
            P = torch.einsum("qa,qb,qzyx->abzyx", self.E, self.E, f[: self.q])
            P = P - j[:, None] * j[None, :]
            eye = torch.eye(3, device="cuda", dtype=torch.float64)
            if not self.three:
                eye[2, 2] = 0
            P = P - eye[:, :, None, None, None] * rho / 3
            v = (2 * self.porosity(g) * (j * j).sum(0)
                 + 4.5 * nu * c.omega ** 2 * (P * P).sum((0, 1))).sum()
        else:
            T = f[self.q:].sum(0)
            if o == G.OBJ_HEAT_FLUX:
                v = -(box(c.obj_out, j[0]) * box(c.obj_out, T)).sum()
            elif o == G.OBJ_DOMAIN_TEMPERATURE:
                v = box(c.obj_out, T).mean()
            else:
                ti, tb = c.obj_param[0], c.obj_param[1]
                gb, Tb = box(c.obj_out, g), box(c.obj_out, T)
                v = ((1 - gb) * (Tb - ti)).sum() / ((1 - gb) * (tb - ti)).sum()
        return c.obj_weight * v

    def run(self, g, steps):
        f, js = self.start(), []
        for t in range(steps):
            f = self.step(f, g, t)
            js.append(self.objective(f, g))
        return f, torch.stack(js)

    def gradient(self, g, steps, steady=None):
        """J, dJ/dgamma and the steady steps: states kept every `every` steps and
        recomputed in between, each step differentiated by itself."""
        f, t, S, t0 = self.start(), 0, 0, None
        every = max(1, int(math.isqrt(steps + (steady[0] if steady else 0))))
        kept = {0: f}
        with torch.no_grad():
            if steady:
                most, check, tol = steady
                while S < most:
                    p, f = f, self.step(f, g, t)
                    t += 1
                    S += 1
                    if t % every == 0:
                        kept[t] = f
                    if (S % check == 0 or S == most) and float((f - p).abs().max()) < tol:
                        break
                t0 = S
            while t < S + steps:
                f = self.step(f, g, t, t0)
                t += 1
                if t % every == 0:
                    kept[t] = f
        n, J = t, 0.0
        dg, lam, block = torch.zeros_like(g), None, {n: f}
        for t in range(n, -1, -1):
            if t not in block:
                block, s = {}, t // every * every
                v = kept[s]
                with torch.no_grad():
                    while s < t:
                        block[s] = v
                        v = self.step(v, g, s, t0 if s >= S else None)
                        s += 1
                block[t] = v
            with torch.enable_grad():
                x = block.pop(t).detach().requires_grad_()
                y = g.detach().requires_grad_()
                total = 0.0
                if lam is not None:
                    total = (lam * self.step(x, y, t, t0 if t >= S else None)).sum()
                if t > S:
                    F = self.objective(x, y)
                    total = total + F
                    J += float(F.detach())
                lam, d = torch.autograd.grad(total, (x, y), allow_unused=True)
            if d is not None:
                dg += d
        return J, dg, S


def _pull_cells(f):
    """(Q, nz, ny, nx) -> cell-major order, as populations() returns it."""
    return f.reshape(f.shape[0], -1).t().contiguous().reshape(-1).cpu().numpy()


def _gamma_torch(cfg, gamma):
    return torch.from_numpy(gamma).cuda().reshape(cfg.nz if cfg.lattice == G.D3Q19 else 1,
                                                  cfg.ny, cfg.nx)


def _filter_taps(rad, three):
    r = range(-rad, rad + 1)
    taps = []
    for dz in (r if three else [0]):
        for dy in r:
            for dx in r:
                d = math.sqrt(dx * dx + dy * dy + dz * dz)
                if d < rad:
                    taps.append((dz, dy, dx, rad - d))
    return taps


def _filter(x, box, rad, beta, eta):
    """Cone filter on the rows of the box (weights rad - distance, neighbours
    inside the grid, divided by the row sum), then the tanh projection there."""
    taps = _filter_taps(rad, x.shape[0] > 1)
    pad = (rad, rad, rad, rad) + ((rad, rad) if x.shape[0] > 1 else (0, 0))
    xp = torch.nn.functional.pad(x, pad)
    op = torch.nn.functional.pad(torch.ones_like(x), pad)
    z0 = rad if x.shape[0] > 1 else 0
    acc, den = torch.zeros_like(x), torch.zeros_like(x)
    for dz, dy, dx, w in taps:
        at = (slice(z0 + dz, z0 + dz + x.shape[0]), slice(rad + dy, rad + dy + x.shape[1]),
              slice(rad + dx, rad + dx + x.shape[2]))
        acc = acc + w * xp[at]
        den = den + w * op[at]
    v = acc / den
    v = (math.tanh(beta * eta) + torch.tanh(beta * (v - eta))) / (
        math.tanh(beta * eta) + math.tanh(beta * (1 - eta)))
    m = torch.zeros_like(x, dtype=torch.bool)
    m[box[4]:box[5] + 1, box[2]:box[3] + 1, box[0]:box[1] + 1] = True
    return torch.where(m, v, x)


def _exact_design(case, seed):
    box, stages, etas, n = _design_update(case)
    x, sens = _design_inputs(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    out = {"gamma": [], "dJdx": [], "change": None, "constraints": None, "x": None}
    for r, eta in enumerate(etas):
        v = torch.from_numpy(x).cuda().requires_grad_()
        full = torch.ones(shape, device="cuda", dtype=torch.float64)
        at = (slice(box[4], box[5] + 1), slice(box[2], box[3] + 1), slice(box[0], box[1] + 1))
        full = full.clone()
        full[at] = v.reshape(full[at].shape)
        for k, (rad, _, beta, e) in enumerate(stages):
            last = k == len(stages) - 1 and len(etas) > 1
            full = _filter(full, box, rad, beta, eta if last else e)
        s = torch.from_numpy(sens[r][1]).cuda().reshape(shape)
        (d,) = torch.autograd.grad((full * s).sum(), v)
        out["gamma"].append(full.detach().reshape(-1).cpu().numpy())
        out["dJdx"].append(d.cpu().numpy())
    return out


# the most that exact() works through: cells times steps times populations
MOST_EXACT = 3.5e10


def exact(case, seed):
    kind = case["kind"]
    if kind == "design":
        taps = sum((2 * s + 1) ** (3 if case["nz"] > 1 else 2) for s in (case["radius"],
                                                                       case["radius2"]))
        if taps * case["nx"] * case["ny"] * case["nz"] > 1.2e9:
            return None   # the saved products of every tap would not fit
        return _exact_design(case, seed)
    grids = _batch_grids(case) if kind == "batch" else [(case["nx"], case["ny"])]
    cells = sum(a * b for a, b in grids) * case["nz"]
    steps = case["steps"] + case.get("max_steady", 0)
    calls = steps * len(grids) * (1 if kind in ("forward", "stepwise") else 4)
    if cells * steps * NPOP[LATTICES[case["model"]]] > MOST_EXACT or calls > 10000:
        return None
    if kind == "batch":
        out = {"J": [], "dJdgamma": [], "recomputed": None}
        for k, (nx, ny) in enumerate(grids):
            cfg = _config(case, nx, ny)
            J, d, _ = _Model(cfg).gradient(
                _gamma_torch(cfg, _design(case["model"], nx, ny, 1, seed, k)), case["steps"])
            out["J"].append(J)
            out["dJdgamma"].append(d.reshape(-1).cpu().numpy())
        out["J"] = np.array(out["J"])
        return out
    cfg = _config(case)
    table = W.pump_inflow_profile(cfg) if case["model"] == "pump" else None
    g = _gamma_torch(cfg, _design(case["model"], case["nx"], case["ny"], case["nz"], seed))
    m = _Model(cfg, table)
    if kind in ("stepwise", "forward"):
        with torch.no_grad():
            f, js = m.run(g, case["steps"])
            rho, j = m.macros(f)
            mac = torch.cat([rho[None], j if m.three else j[:2]])
            if m.heat:
                mac = torch.cat([mac, f[m.q:].sum(0)[None]])
        out = {"macros": _pull_cells(mac), "populations": _pull_cells(f)}
        if kind == "stepwise":
            return {"J": js.cpu().numpy(), **out}
        return {"J": float(js.sum()), "steps": js.cpu().numpy(), **out}
    if kind == "steady":
        J, d, _ = m.gradient(g, case["steps"], (case["max_steady"], case["check"], 1e-7))
        return {"J": J, "dJdgamma": d.reshape(-1).cpu().numpy(), "steady": None,
                "recomputed": None}
    J, d, _ = m.gradient(g, case["steps"])
    return {"J": J, "dJdgamma": d.reshape(-1).cpu().numpy(), "recomputed": None}
