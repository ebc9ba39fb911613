"""The workloads whose speed this repository is held to, each one pass through
its public entry points, with inputs made from a seed and, where one exists in
reasonable time, the result in 64-bit arithmetic.

A pass is one of
  step       EdgeSim.step(), the whole substep a driver runs per time step
  march      one backward-map march on the packed map the device driver keeps
  dropin     the EDGE march through the reference's own signature
  advect     the semi-Lagrangian half step of the face velocity
  transport  forward map, velocity and dye pullback through it, and the clamp
  backtrack  the EFM backward map through the cached velocities
  project    the pressure projection (plain walls)
  solid      the pressure projection around a solid obstacle
  particles  the laden-particle kernels of one step (gather, update, scatter)
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "edge-flow-maps_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

WALLS = ((2, 2), (2, 2), (2, 2))
CFL = 0.5
EPS_FRAC = 0.025  # epsilon of the epsilon-difference marches, in cells
REINIT = 12       # steps between reinitialisations of the flow map
VARIANT = {"edge": 1, "ed4": 0, "ed8": 2}


def listed():
    return [
        # the smallest whole step: the 64x32x32 leapfrogging configuration, where launches and the host loop count
        dict(name="step_64x32x32", kind="step", variant="edge", nx=64, ny=32, nz=32),
        # the headline configuration: the EDGE step at 256x128x128
        dict(name="step_256x128x128", kind="step", variant="edge", nx=256, ny=128, nz=128),
        # a user of the reference's hermite.py: the EDGE march in its layout, in place
        dict(name="dropin_edge_128x64x64", kind="dropin", nx=128, ny=64, nz=64),
        # the ED4 march on a ragged grid whose spacing is no power of two
        dict(name="march_ed4_100x75x61", kind="march", variant="ed4", nx=100, ny=75, nz=61),
        # the ED8 march at the size of the four-vortex case
        dict(name="march_ed8_128x128x256", kind="march", variant="ed8", nx=128, ny=128, nz=256),
        # the half step of the velocity on a small odd grid
        dict(name="advect_97x65x49", kind="advect", nx=97, ny=65, nz=49),
        # forward map and pullbacks at an ordinary size
        dict(name="transport_192x96x96", kind="transport", nx=192, ny=96, nz=96),
        # EFM's backward map half way through a reinitialisation interval
        dict(name="backtrack_128x64x64", kind="backtrack", nx=128, ny=64, nz=64, steps=6),
        # a projection of the headline size, which the caches hold
        dict(name="project_256x128x128", kind="project", nx=256, ny=128, nz=128, base_level=2, precision=0),
        # the largest projection: 33.5 M cells, bound by memory
        dict(name="project_512x256x256", kind="project", nx=512, ny=256, nz=256, base_level=2, precision=0),
        # the delta-wing case: a wedge and a moving shell in a 256x128x128 box
        dict(name="solid_256x128x128", kind="solid", nx=256, ny=128, nz=128, base_level=3),
        # the ink-circle case: a million laden particles in a 128x256x128 box
        dict(name="particles_1m", kind="particles", nx=128, ny=256, nz=128, num=1000000),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi, cells):
        while True:
            n = [size(lo, hi) for _ in range(3)]
            if n[0] * n[1] * n[2] <= cells:
                return dict(nx=n[0], ny=n[1], nz=n[2])

    def levels(lo, hi, cells, base_level):
        # a grid that halves exactly on every level of its multigrid pyramid
        while True:
            mn = 8 * rng.randint(lo // 8, hi // 8)
            unit = 2 ** max(0, int(math.log2(mn)) - base_level)
            if mn % unit == 0:
                n = [mn, unit * rng.randint(mn // unit, 2 * mn // unit), mn]
                n[rng.randint(0, 1)] = unit * rng.randint(mn // unit, 4 * mn // unit)
                if n[0] * n[1] * n[2] <= cells:
                    return dict(nx=n[0], ny=n[1], nz=n[2])

    kind = rng.choice(["step", "march", "march", "dropin", "advect", "transport", "backtrack", "project", "solid",
                       "particles"])
    c = dict(kind=kind)
    if kind == "step":
        c.update(variant=rng.choice(["edge", "edge", "ed4", "ed8", "ge", "efm"]), **levels(32, 128, 256 * 128 * 96, 2))
    elif kind == "march":
        c.update(variant=rng.choice(["edge", "edge", "ed4", "ed8", "ge"]), **grid(24, 256, 256 * 128 * 128))
    elif kind == "dropin":
        c.update(grid(24, 256, 2 * 128 * 128 * 64))
    elif kind in ("advect", "transport"):
        c.update(grid(24, 300, 256 * 128 * 128))
    elif kind == "backtrack":
        c.update(grid(24, 160, 128 * 128 * 64), steps=rng.randint(1, REINIT))
    elif kind == "project":
        c.update(levels(32, 192, 384 * 192 * 192, 2), base_level=2, precision=rng.choice([0, 0, 2]))
    elif kind == "solid":
        # room for the wedge, a chord long, between the walls
        ny = 16 * rng.randint(2, 8)
        unit = 2 ** (int(math.log2(ny)) - 3)
        ny -= ny % unit
        c.update(nx=unit * rng.randint(-(-3 * ny // (2 * unit)), 2 * ny // unit), ny=ny, nz=ny, base_level=3)
    else:
        c.update(grid(32, 256, 256 * 128 * 128), num=size(20000, 4000000))
    return c


def _res(c):
    return int(c["nx"]), int(c["ny"]), int(c["nz"])


def _dx(c):
    """Grid spacing: the particle cases count length in cells, the others in
    units of the shorter cross-section axis, as the drivers do."""
    return 1.0 if c["kind"] == "particles" else 1.0 / min(c["ny"], c["nz"])


# -- inputs -------------------------------------------------------------------
# Smooth vector fields whose normal component vanishes on the walls of the box:
# component d is a sum of modes, sin along d and cos along the other two axes.
class _Modes:
    def __init__(self, res, dx, rng, count=14, kmax=5, divfree=True):
        L = [n * dx for n in res]
        m = rng.integers(1, kmax + 1, size=(count, 3))
        self.k = np.pi * m / np.asarray(L)  # (M, 3)
        a = rng.standard_normal((count, 3)) * (np.linalg.norm(m, axis=1) ** -1.8)[:, None]
        if divfree:
            a = a - self.k * ((a * self.k).sum(1) / (self.k ** 2).sum(1))[:, None]
        self.a = a

    def field(self, comp, axes, der=(0, 0, 0)):
        """Component `comp` (differentiated der[d] times along d) at the tensor
        grid of the three coordinate vectors `axes`, float64 on the GPU."""
        f, amp = [], np.array(self.a[:, comp])
        for d in range(3):
            x = torch.as_tensor(axes[d], dtype=torch.float64, device="cuda")
            ph = torch.as_tensor(self.k[:, d], device="cuda")[:, None] * x[None, :]
            s = d == comp  # sin along the component's own axis
            if der[d]:
                amp = amp * self.k[:, d] * (1.0 if s else -1.0)
                s = not s
            f.append(torch.sin(ph) if s else torch.cos(ph))
        n = [t.shape[1] for t in f]
        left = torch.einsum("mi,mj->ijm", f[0] * torch.as_tensor(amp, device="cuda")[:, None], f[1])
        return (left.reshape(n[0] * n[1], -1) @ f[2]).reshape(n)


def _cells(res, dx):
    return [(np.arange(n) + 0.5) * dx for n in res]


def _faces(res, dx, a):
    return [np.arange(n + 1) * dx if d == a else (np.arange(n) + 0.5) * dx for d, n in enumerate(res)]


def _velocity(res, dx, rng, divfree=True, rough=0.0):
    """Face velocities of maximum speed 1 (plus seeded noise of relative size
    `rough`, what a step leaves before its projection)."""
    M = _Modes(res, dx, rng, divfree=divfree)
    u = [M.field(d, _faces(res, dx, d)) for d in range(3)]
    s = 1.0 / max(float(t.abs().max()) for t in u)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 31)))
    out = []
    for t in u:
        t = t * s
        if rough:
            t = t + rough * torch.randn(t.shape, generator=g, device="cuda", dtype=torch.float64)
        out.append(t.float().contiguous())
    return out


def _dye(res, dx, rng):
    X = [torch.as_tensor(x, device="cuda") for x in _cells(res, dx)]
    out = torch.zeros(tuple(res) + (4,), dtype=torch.float32, device="cuda")
    for ch in range(4):
        c = [float(rng.uniform(0.25, 0.75)) * n * dx for n in res]
        r = 0.2 * min(res) * dx
        d2 = sum(((x - cc) ** 2).reshape([-1 if q == d else 1 for q in range(3)])
                 for d, (x, cc) in enumerate(zip(X, c)))
        out[..., ch] = torch.exp(-d2 / (r * r)).float()
    return out.contiguous()


def _map(res, dx, rng):
    """A backward map some steps after its reset: psi = X + a displacement of a
    few cells, with its exact gradient and mixed derivatives, in the
    reference's layout (psi, rows T_c, (yz, xz, xy) rows dT_c, d2T_c)."""
    M = _Modes(res, dx, rng)
    ax = _cells(res, dx)
    D = [M.field(c, ax) for c in range(3)]
    s = 2.0 * dx / max(float(t.abs().max()) for t in D)
    X = torch.meshgrid(*[torch.as_tensor(x, device="cuda") for x in ax], indexing="ij")
    psi = torch.stack([X[c] + s * D[c] for c in range(3)], -1).float().contiguous()
    T, dT, d2T = [], [], []
    for c in range(3):
        g = [s * M.field(c, ax, tuple(int(d == e) for e in range(3))) + (1.0 if c == d else 0.0) for d in range(3)]
        T.append(torch.stack(g, -1).float().contiguous())
        h = [s * M.field(c, ax, der) for der in ((0, 1, 1), (1, 0, 1), (1, 1, 0))]
        dT.append(torch.stack(h, -1).float().contiguous())
        d2T.append((s * M.field(c, ax, (1, 1, 1))).float().contiguous())
    return psi, T, dT, d2T


def _particles(c, rng):
    res, dx, n = _res(c), _dx(c), int(c["num"])
    L = np.array([r * dx for r in res])
    # a drop of radius 0.18 of the narrowest axis around the middle
    p = rng.standard_normal((n, 3))
    p = p / np.linalg.norm(p, axis=1)[:, None] * (rng.random(n) ** (1 / 3))[:, None] * 0.18 * L.min() + L * 0.5
    v = 0.2 * rng.standard_normal((n, 3))
    rad = 0.005 + 0.005 * rng.random(n)
    cu = lambda a: torch.as_tensor(a.astype(np.float32), device="cuda").contiguous()  # noqa: E731
    return cu(p), cu(v), cu(rad), [float(x) for x in L]


LP = dict(Re=5.5, St=6.6e-2, gravity=1.0, density_ratio=2.0 / 3, erad=35.0, lrad=0.01)


def prepare(case, seed):
    from edgeb200 import ops
    from edgeb200.fields import zeros_cells, zeros_faces
    rng = np.random.default_rng(int(seed))
    res, dx, kind = _res(case), _dx(case), case["kind"]
    s = {"case": case, "res": res, "dx": dx, "dt": CFL * dx, "pass": 0}
    if kind == "step":
        from edgeb200.sim import EdgeSim
        sim = EdgeSim(res, dx, variant=case["variant"], cfl=CFL, reinit_every=REINIT, ed_eps=EPS_FRAC * dx,
                      base_level=2)
        sim.set_velocity(*_velocity(res, dx, rng))
        sim.set_smoke(_dye(res, dx, rng))
        s["sim"] = sim
    elif kind == "march":
        hv = 2 if case["variant"] == "ge" else VARIANT[case["variant"]]
        m = _map(res, dx, rng)
        s["hv"], s["u"] = hv, _velocity(res, dx, rng)
        s["src"], s["dst"] = (torch.zeros((ops.PLANES[hv],) + res + (4,), device="cuda") for _ in range(2))
        ops.map_pack(hv, *m[:2], m[2] if hv else None, m[3] if hv == 2 else None, s["src"])
    elif kind == "dropin":
        s["u"] = _velocity(res, dx, rng)
        v3 = lambda: zeros_cells(res, 3)  # noqa: E731
        s["map"], s["tmp"] = [v3() for _ in range(7)], [v3() for _ in range(7)]
        s["X"] = torch.stack(torch.meshgrid(*[torch.as_tensor(x, device="cuda") for x in _cells(res, dx)],
                                            indexing="ij"), -1).float().contiguous()
    elif kind == "advect":
        s["u"], s["u1"] = _velocity(res, dx, rng), zeros_faces(res)
    elif kind == "transport":
        s["u"], s["u0"] = _velocity(res, dx, rng), _velocity(res, dx, rng)
        s["dye0"], s["dye"] = _dye(res, dx, rng), zeros_cells(res, 4)
        s["phi"], s["F"], s["u1"], s["u2"] = zeros_faces(res, 3), zeros_faces(res, 3), zeros_faces(res), \
            zeros_faces(res)
    elif kind == "backtrack":
        s["cache"] = [_velocity(res, dx, rng) for _ in range(int(case["steps"]))]
        s["dts"] = [CFL * dx * float(rng.uniform(0.7, 1.0)) for _ in s["cache"]]
        s["psi"], s["T"] = zeros_faces(res, 3), zeros_faces(res, 3)
    elif kind == "project":
        from sim.mgpcg import MGPCG_3
        s["u0"] = _velocity(res, dx, rng, divfree=False, rough=0.02)
        s["u"] = [torch.empty_like(t) for t in s["u0"]]
        if case["precision"]:
            from edgeb200.projection import Projection
            s["proj"] = Projection(res, base_level=case["base_level"], precision=case["precision"])
        else:
            s["solver"] = MGPCG_3(WALLS, list(res), base_level=case["base_level"])
    elif kind == "solid":
        from edgeb200.sim import wedge_mask
        from sim.mgpcg_solid import MGPCG_Solid_3
        # the wind of the delta-wing case and a disturbance
        wind = (0.6 * math.cos(math.radians(20)), 0.0, 0.6 * math.sin(math.radians(20)))
        s["u0"] = [w + 0.1 * t for w, t in zip(wind, _velocity(res, dx, rng, divfree=False, rough=0.02))]
        s["u"] = [torch.empty_like(t) for t in s["u0"]]
        mask, bvel = wedge_mask(res, dx)
        s["solver"] = MGPCG_Solid_3(WALLS, mask, bvel, list(res), base_level=case["base_level"])
    else:
        s["u"] = _velocity(res, dx, rng)
        s["pos0"], s["vel0"], s["rad"], s["L"] = _particles(case, rng)
        for k in ("pos", "vel", "acc", "vdiff"):
            s[k] = torch.zeros_like(s["pos0"])
        s["drag"], s["vis"] = zeros_faces(res), zeros_faces(res)
    return s


def run(s):
    from edgeb200 import ops
    case, res, dx, dt = s["case"], s["res"], s["dx"], s["dt"]
    kind, at = case["kind"], s["pass"]
    s["pass"] = at + 1
    if kind == "step":
        sim = s["sim"]
        sim.step()
        out = {"u": list(sim.u), "dye": sim.smoke, "phi": list(sim.phi), "F": list(sim.F)}
        if sim.variant != "efm":
            out["map"] = sim.pmaps[sim.cur]
        return out
    if kind == "march":
        if case["variant"] == "ge":
            ops.march_ge_packed(s["u"], dx, dt, s["src"], s["dst"], res)
        else:
            ops.march_packed(s["hv"], s["u"], dx, dt, EPS_FRAC * dx, s["src"], s["dst"], res)
        return list(s["dst"])
    if kind == "dropin":
        from sim import hermite
        if at % REINIT == 0:
            hermite.reset_to_identity_2(*s["map"], s["X"])
        hermite.advect_psi_garm_ed4_fusion_unroll(*s["tmp"], *s["map"], *s["u"], s["X"], dx, dt, EPS_FRAC * dx)
        return s["map"]
    if kind == "advect":
        from sim import hermite
        hermite.advect_u_semi_lagrangian(*s["u"], *s["u1"], dx, 0.5 * dt, None, None, None)
        return s["u1"]
    if kind == "transport":
        if at % REINIT == 0:
            ops.reset_faces(res, dx, s["phi"], s["F"])
        ops.advance_map(s["u"], dx, dt, s["phi"], s["F"])
        ops.pullback_u(s["u0"], dx, s["phi"], s["F"], s["u1"])
        ops.pullback_dye(s["dye0"], dx, s["phi"], s["dye"], init=s["dye0"], scale=0.5)
        ops.clamp_u(s["u1"], s["u0"], s["u2"])
        return {"phi": s["phi"], "F": s["F"], "u1": s["u1"], "u2": s["u2"], "dye": s["dye"]}
    if kind == "backtrack":
        ops.efm_backtrack(s["cache"], s["dts"], dx, s["psi"], s["T"])
        return {"psi": s["psi"], "T": s["T"]}
    if kind in ("project", "solid"):
        # each step hands the solver a new velocity
        for d, a in zip(s["u"], s["u0"]):
            d.copy_(a)
        if "proj" in s:
            s["proj"].poisson(*s["u"])
        else:
            s["solver"].Poisson(*s["u"])
        return s["u"]
    from sim import lp
    n, L, u = int(case["num"]), s["L"], s["u"]
    s["pos"].copy_(s["pos0"])
    s["vel"].copy_(s["vel0"])
    lp.update_particles_acc(*u, s["vel"], s["pos"], s["acc"], dx, dt, n, LP["St"], LP["gravity"])
    lp.update_particles_velocity(s["acc"], s["vel"], s["pos"], dt, dx, n, *L)
    lp.calculate_velocity_diff(*u, s["vel"], s["vdiff"], s["pos"], dx, n, LP["St"], LP["density_ratio"], LP["erad"])
    lp.laden_particles_back_with_computing_particle(*s["drag"], *u, s["vel"], s["vdiff"], s["pos"], s["rad"], dx, n,
                                                    LP["lrad"], *L, *res)
    lp.update_particles_position(s["vel"], s["pos"], dt, n, *L)
    lp.calculate_viscous_force(*u, *s["vis"], dx, LP["Re"])
    return {"acc": s["acc"], "vel": s["vel"], "pos": s["pos"], "vdiff": s["vdiff"], "drag": s["drag"],
            "vis": s["vis"]}


def work(case):
    """Bytes: each input field read once and each output written once.
    Operations: the reference's arithmetic per cell, face or particle."""
    nx, ny, nz = _res(case)
    n, kind = nx * ny * nz, case["kind"]
    f = (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)
    state = {"edge": 84, "ed4": 48, "ed8": 96, "ge": 96, "efm": 0}        # bytes of one map per cell
    march = {"edge": 27400, "ed4": 8400, "ed8": 16800, "ge": 5500, "efm": 18000}
    if kind == "step":
        # u, dye and maps in and out, the interval's initial fields in; a
        # projection reads and writes the velocity
        v = case["variant"]
        return {"bytes": f * (8 + 4 + 48 + 2 * 8) + n * (48 + 2 * state[v]),
                "flops": n * (march[v] + 2 * 4 * 150) + f * (1550 + 3000 + 3 * 330 + 1200)}
    if kind in ("march", "dropin"):
        v = case.get("variant", "edge")
        return {"bytes": 4 * f + 2 * n * state[v], "flops": n * march[v]}
    if kind == "advect":
        return {"bytes": 8 * f, "flops": 1550 * f}
    if kind == "transport":
        return {"bytes": f * (4 + 48 + 4 + 4 + 4) + 32 * n, "flops": f * (3000 + 330) + 100 * n}
    if kind == "backtrack":
        return {"bytes": f * (4 * case["steps"] + 24), "flops": 3000 * f * case["steps"]}
    if kind in ("project", "solid"):
        return {"bytes": 8 * f + (4 * n if kind == "solid" else 0), "flops": n * 150 * (4 if kind == "project" else 9)}
    p = int(case["num"])
    return {"bytes": p * (12 * 3 + 4 + 12 * 4) + f * 12, "flops": p * 3 * 350 + 10 * f}


# -- the same results in 64 bits ------------------------------------------------
_f = lambda x: float(np.float32(x))  # noqa: E731  the entry points take float32 scalars
_ED4 = ((-1, -1, -1), (1, 1, -1), (-1, 1, 1), (1, -1, 1))
_ED8 = ((-1, -1, -1), (1, -1, -1), (-1, 1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, 1), (1, 1, 1))


def _bound(n, minus):
    return _f(float(n - minus) - 1e-6)


def _spline(f, a, p, dx, grad):
    """Quadratic B-spline of the face field f (normal axis a) at points p (N, 3):
    value (N,) and gradient (N, 3)."""
    idx, w, dw = [], [], []
    for d in range(3):
        s = (p[:, d] / dx - (0.0 if d == a else 0.5)).clamp(1.0, _bound(f.shape[d], 2))
        b = torch.floor(s - 0.5)
        x = s - b
        idx.append(b.long())
        w.append((0.5 * (1.5 - x) ** 2, 0.75 - (x - 1) ** 2, 0.5 * (x - 0.5) ** 2))
        dw.append((x - 1.5, -2 * (x - 1), x - 0.5))
    flat, (n1, n2) = f.reshape(-1), f.shape[1:]
    v = torch.zeros_like(p[:, 0])
    g = [torch.zeros_like(v) for _ in range(3)] if grad else None
    for i in range(3):
        for j in range(3):
            row = ((idx[0] + i) * n1 + idx[1] + j) * n2 + idx[2]
            q = [flat[row + k] for k in range(3)]
            c = w[2][0] * q[0] + w[2][1] * q[1] + w[2][2] * q[2]
            v += w[0][i] * w[1][j] * c
            if grad:
                g[0] += dw[0][i] * w[1][j] * c
                g[1] += w[0][i] * dw[1][j] * c
                g[2] += w[0][i] * w[1][j] * (dw[2][0] * q[0] + dw[2][1] * q[1] + dw[2][2] * q[2])
    return v, torch.stack(g, -1) / dx if grad else None


def _sample(u, p, dx, grad=False):
    r = [_spline(u[a], a, p, dx, grad) for a in range(3)]
    return torch.stack([x[0] for x in r], -1), torch.stack([x[1] for x in r], 1) if grad else None


def _rk4(u, p, C, dt, dx):
    """RK4 of points p (N, 3) and, if given, Jacobian columns C (N, 3, m)."""
    k, kc, q, Q = [], [], p, C
    for st in range(4):
        v, G = _sample(u, q, dx, C is not None)
        k.append(v)
        if C is not None:
            kc.append(G @ Q)
        h = (0.5 * dt, 0.5 * dt, dt, 0.0)[st]
        q = p + h * v
        Q = C + h * kc[-1] if C is not None else None
    p = p + dt / 6 * (k[0] + 2 * k[1] + 2 * k[2] + k[3])
    return p, (C + dt / 6 * (kc[0] + 2 * kc[1] + 2 * kc[2] + kc[3]) if C is not None else None)


def _shift(t, d, step):
    n = t.shape[d]
    return t.index_select(d, (torch.arange(n, device=t.device) + step).clamp(0, n - 1))


def _diff(t, d):
    return _shift(t, d, 1) - _shift(t, d, -1)


def _coefs(hv, psi, g, h, t3, dx):
    """The 8 Hermite coefficient fields per cell, bit 0/1/2 of the index = the
    g basis along x/y/z; psi (.., 3), g[d] and h = (yz, xz, xy) columns."""
    if hv == 0:
        h = [(_diff(g[1], 2) + _diff(g[2], 1)) / 4 / dx, (_diff(g[0], 2) + _diff(g[2], 0)) / 4 / dx,
             (_diff(g[0], 1) + _diff(g[1], 0)) / 4 / dx]
        sh = lambda t, *m: [t := _shift(t, d, s) for d, s in m][-1]  # noqa: E731
        v30 = _diff(sh(g[1], (0, 1)), 2) + _diff(sh(g[2], (0, 1)), 1)
        v31 = _diff(sh(g[1], (0, -1)), 2) + _diff(sh(g[2], (0, -1)), 1)
        v32 = _diff(sh(g[0], (1, 1)), 2) + _diff(sh(g[2], (1, 1)), 0)
        v33 = _diff(sh(g[0], (1, -1)), 2) + _diff(sh(g[2], (1, -1)), 0)
        v34 = _diff(sh(g[0], (2, 1)), 1) + _diff(sh(g[1], (2, 1)), 0)
        v35 = _diff(sh(g[0], (2, -1)), 1) + _diff(sh(g[1], (2, -1)), 0)
        t3 = (v30 - v31 + v32 - v33 + v34 - v35) / 24 / dx ** 2
    elif hv == 1:
        t3 = (_diff(h[0], 0) + _diff(h[1], 1) + _diff(h[2], 2)) / 6 / dx
    return {0: psi, 1: g[0] * dx, 2: g[1] * dx, 4: g[2] * dx, 6: h[0] * dx ** 2, 5: h[1] * dx ** 2,
            3: h[2] * dx ** 2, 7: t3 * dx ** 3}


def _hermite(co, p, dx, grad):
    shp = co[0].shape[:3]
    B = []
    for d in range(3):
        s = (p[:, d] / dx - 0.5).clamp(1.0, _bound(shp[d], 2))
        b = torch.floor(s)
        f = []
        for i in range(2):
            x = s - b - i
            a, sg = x.abs(), torch.where(x < 0, -1.0, 1.0)
            f.append((2 * a ** 3 - 3 * a ** 2 + 1, sg * (a ** 3 - 2 * a ** 2 + a), sg * (6 * a ** 2 - 6 * a),
                      3 * a ** 2 - 4 * a + 1))
        B.append((b.long(), f))
    val = torch.zeros((p.shape[0], 3), dtype=torch.float64, device=p.device)
    G = torch.zeros((p.shape[0], 3, 3), dtype=torch.float64, device=p.device) if grad else None
    for i in range(2):
        for j in range(2):
            for k in range(2):
                at = [(B[d][0] + o).clamp(max=shp[d] - 1) for d, o in enumerate((i, j, k))]
                e = (at[0] * shp[1] + at[1]) * shp[2] + at[2]
                for b in range(8):
                    c = co[b].reshape(-1, 3)[e]
                    w = [B[d][1][o] for d, o in enumerate((i, j, k))]
                    q = [(b >> d) & 1 for d in range(3)]
                    f = [w[d][q[d]] for d in range(3)]
                    val += (f[0] * f[1] * f[2])[:, None] * c
                    if grad:
                        h = [w[d][2 + q[d]] for d in range(3)]
                        for d in range(3):
                            t = f[:d] + [h[d]] + f[d + 1:]
                            G[:, :, d] += (t[0] * t[1] * t[2])[:, None] * c / dx
    return val, G


def _centres(res, dx, lo, hi):
    e = torch.arange(lo, hi, device="cuda")
    return torch.stack([e // (res[1] * res[2]), e // res[2] % res[1], e % res[2]], -1).double().add_(0.5).mul_(dx)


def _march64(variant, res, dx, dt, eps, u, psi, g, h, t3):
    """The marched packed map (8, nx, ny, nz, 4) in float64."""
    hv = {"edge": 1, "ed4": 0, "ed8": 2, "ge": 2}[variant]
    co = _coefs(hv, psi, g, h, t3, dx)
    n = res[0] * res[1] * res[2]
    out = torch.zeros((8, n, 4), dtype=torch.float64, device="cuda")
    for lo in range(0, n, 1 << 20):
        hi = min(n, lo + (1 << 20))
        X = _centres(res, dx, lo, hi)
        off = lambda o: X + torch.tensor(o, dtype=torch.float64, device="cuda") * eps  # noqa: E731
        o = out[:, lo:hi, :3]
        if variant in ("edge", "ge"):
            I3 = torch.eye(3, dtype=torch.float64, device="cuda").expand(hi - lo, 3, 3)
            for q, of in enumerate(((0, 0, 0),) + (_ED4 if variant == "edge" else ())):
                P, C = _rk4(u, off(of), I3, -dt, dx)
                v, G = _hermite(co, P, dx, True)
                T = G @ C
                if q == 0:
                    o[0] = v
                    for d in range(3):
                        o[1 + d] = T[:, :, d]
                else:
                    sx, sy, sz = of
                    o[4] += (sz * T[:, :, 1] + sy * T[:, :, 2]) / 8 / eps
                    o[5] += (sz * T[:, :, 0] + sx * T[:, :, 2]) / 8 / eps
                    o[6] += (sy * T[:, :, 0] + sx * T[:, :, 1]) / 8 / eps
        else:
            pts = _ED4 if variant == "ed4" else _ED8
            for of in pts:
                P = _hermite(co, _rk4(u, off(of), None, -dt, dx)[0], dx, False)[0]
                sx, sy, sz = of
                m = len(pts)
                o[0] += P / m
                for d in range(3):
                    o[1 + d] += of[d] * P / m / eps
                if variant == "ed8":
                    o[4] += sy * sz * P / m / eps ** 2
                    o[5] += sx * sz * P / m / eps ** 2
                    o[6] += sx * sy * P / m / eps ** 2
                    o[7] += sx * sy * sz * P / m / eps ** 3
    out = out.reshape((8,) + tuple(res) + (4,))
    v = [out[q, ..., :3] for q in range(8)]
    if variant == "edge":  # the derived plane: the triple coefficient before its scaling by dx^2
        out[7, ..., :3] = (_diff(v[4], 0) + _diff(v[5], 1) + _diff(v[6], 2)) / 6
    elif variant == "ed4":  # the derived planes, before their scaling by dx
        c = _coefs(0, v[0], v[1:4], None, None, dx)
        for q, b in ((4, 6), (5, 5), (6, 3), (7, 7)):
            out[q, ..., :3] = c[b] / dx
    elif variant == "ge":
        out[4, ..., :3] = (_diff(v[2], 2) + _diff(v[3], 1)) / 4 / dx
        out[5, ..., :3] = (_diff(v[1], 2) + _diff(v[3], 0)) / 4 / dx
        out[6, ..., :3] = (_diff(v[1], 1) + _diff(v[2], 0)) / 4 / dx
        out[7, ..., :3] = (_diff(v[4], 0) + _diff(v[5], 1) + _diff(v[6], 2)) / 6 / dx
    return out


def _face_points(res, dx, a):
    return torch.stack(torch.meshgrid(*[torch.as_tensor(x, dtype=torch.float64, device="cuda")
                                        for x in _faces(res, dx, a)], indexing="ij"), -1).reshape(-1, 3)


def _trilinear(f, p, dx):
    idx, w = [], []
    for d in range(3):
        s = (p[:, d] / dx - 0.5).clamp(1.0, _bound(f.shape[d], 1))
        b = torch.floor(s)
        idx.append((b.long(), (b.long() + 1).clamp(max=f.shape[d] - 1)))
        w.append((1 - (s - b), s - b))
    out = 0.0
    for i in range(2):
        for j in range(2):
            for k in range(2):
                e = (idx[0][i] * f.shape[1] + idx[1][j]) * f.shape[2] + idx[2][k]
                out = out + f.reshape(-1, 4)[e] * (w[0][i] * w[1][j] * w[2][k])[:, None]
    return out


def _project64(u, res):
    """Subtract the gradient of the solution of the Neumann problem, which the
    cosine transform diagonalises."""
    for a in range(3):
        u[a].select(a, 0).zero_()
        u[a].select(a, res[a]).zero_()
    b = sum(torch.diff(u[a], dim=a) for a in range(3))
    Q, lam = [], 0.0
    for d, n in enumerate(res):
        k = torch.arange(n, device="cuda", dtype=torch.float64)
        q = torch.cos(math.pi / n * k[:, None] * (k[None, :] + 0.5)) * math.sqrt(2.0 / n)
        q[0] /= math.sqrt(2.0)
        Q.append(q)
        lam = lam + (2 * torch.cos(math.pi / n * k) - 2).reshape([-1 if e == d else 1 for e in range(3)])
    t = torch.einsum("ai,ijk->ajk", Q[0], b)
    t = torch.einsum("bj,ajk->abk", Q[1], t)
    t = torch.einsum("ck,abk->abc", Q[2], t)
    lam[0, 0, 0] = 1.0
    t = t / lam
    t[0, 0, 0] = 0.0
    p = torch.einsum("ai,ajk->ijk", Q[0], t)
    p = torch.einsum("bj,ibk->ijk", Q[1], p)
    p = torch.einsum("ck,ijc->ijk", Q[2], p)
    for a in range(3):
        u[a].narrow(a, 1, res[a] - 1).sub_(torch.diff(p, dim=a))
    return u


def _particles64(s, case, res, dx, dt):
    u, L = [t.double() for t in s["u"]], s["L"]
    pos, vel, rad = s["pos0"].double(), s["vel0"].double(), s["rad"].double()
    St, grav, lrad = _f(LP["St"]), _f(LP["gravity"]), _f(LP["lrad"])
    at = lambda p: torch.cat([_sample(u, c, dx)[0] for c in p.split(1 << 20)])  # noqa: E731
    v = at(pos)
    acc = -(vel - v) / St
    acc[:, 1] += grav
    acc = acc / (1 + dt / St)
    vel = vel + acc * dt
    lo, hi = (3 * dx, dx, 3 * dx), [x - 3 * dx for x in L]
    for d in range(3):
        stop = ((pos[:, d] < lo[d]) & (vel[:, d] < 0)) | ((pos[:, d] > hi[d]) & (vel[:, d] > 0))
        vel[:, d] = torch.where(stop, 0.0, vel[:, d])
    vdiff = (vel - v) / St * _f(LP["density_ratio"]) / _f(LP["erad"]) ** 3
    keep = torch.ones(pos.shape[0], dtype=torch.bool, device="cuda")
    for d in range(3):
        keep &= (pos[:, d] >= 3 * dx) & (pos[:, d] <= hi[d])
    scale, drag = (rad / lrad) ** 3, []
    for a in range(3):
        out = torch.zeros_like(u[a])
        n1, n2 = out.shape[1:]
        q = [pos[keep, d] / dx - (0.0 if d == a else 0.5) for d in range(3)]
        b = [torch.floor(t - 0.5) for t in q]
        w = []
        for d in range(3):
            x = q[d] - b[d]
            w.append((0.5 * (1.5 - x) ** 2, 0.75 - (x - 1) ** 2, 0.5 * (x - 0.5) ** 2))
        val = vdiff[keep, a] * scale[keep]
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    e = ((b[0].long() + i) * n1 + b[1].long() + j) * n2 + b[2].long() + k
                    out.reshape(-1).index_add_(0, e, val * w[0][i] * w[1][j] * w[2][k])
        drag.append(out)
    pos = pos + vel * dt
    for d in range(3):
        pos[:, d] = pos[:, d].clamp(0.0, L[d])
    vis = [(sum(_shift(t, d, 1) + _shift(t, d, -1) for d in range(3)) - 6 * t) / _f(LP["Re"]) / dx ** 2 for t in u]
    return {"acc": acc, "vel": vel, "pos": pos, "vdiff": vdiff, "drag": drag, "vis": vis}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "solid"):
        return None  # a chain of hundreds of launches; the solid solver stops at a tolerance of its own
    s = prepare(case, seed)
    res, dx, dt = s["res"], _f(s["dx"]), _f(s["dt"])
    eps = _f(EPS_FRAC * s["dx"])
    if kind == "march":
        m = s["src"].double()[..., :3]
        u = [t.double() for t in s["u"]]
        o = _march64(case["variant"], res, dx, dt, eps, u, m[0], [m[1], m[2], m[3]], [m[4], m[5], m[6]], m[7])
        # a quotient of float32 positions by epsilon^2 or epsilon^3 keeps no digits to compare, nor does a
        # second difference of quotients by epsilon
        bad = {"edge": (7,), "ed4": (7,), "ed8": (4, 5, 6, 7), "ge": ()}[case["variant"]]
        return [None if q in bad else o[q] for q in range(8)]
    if kind == "dropin":
        n = res[0] * res[1] * res[2]
        psi = _centres(res, dx, 0, n).reshape(tuple(res) + (3,))
        one = torch.eye(3, dtype=torch.float64, device="cuda")
        g = [one[d].expand(tuple(res) + (3,)) for d in range(3)]
        zero = torch.zeros_like(psi)
        o = _march64("edge", res, dx, dt, eps, [t.double() for t in s["u"]], psi, g, [zero] * 3, None)[..., :3]
        # one step from the identity: its mixed derivatives are of the size of their rounding errors
        return [o[0]] + [torch.stack([o[1 + d, ..., c] for d in range(3)], -1) for c in range(3)] + [None] * 3
    if kind == "advect":
        h, u, out = _f(0.5 * s["dt"]), [t.double() for t in s["u"]], []
        for a in range(3):
            p = torch.cat([_rk4(u, q, None, -h, dx)[0] for q in _face_points(res, dx, a).split(1 << 20)])
            out.append(torch.cat([_spline(u[a], a, q, dx, False)[0] for q in p.split(1 << 20)]).reshape(u[a].shape))
        return out
    if kind in ("transport", "backtrack"):
        back = kind == "backtrack"
        chain = list(zip(s["cache"], s["dts"]))[::-1] if back else [(s["u"], -s["dt"])]
        pos, col = [], []
        for a in range(3):
            P, Cs = [], []
            for p in _face_points(res, dx, a).split(1 << 19):
                C = torch.zeros((p.shape[0], 3, 1), dtype=torch.float64, device="cuda")
                C[:, a] = 1.0
                for u, h in chain:
                    p, C = _rk4([t.double() for t in u], p, C, -_f(h), dx)
                P.append(p)
                Cs.append(C[:, :, 0])
            shape = tuple(n + (d == a) for d, n in enumerate(res)) + (3,)
            pos.append(torch.cat(P).reshape(shape))
            col.append(torch.cat(Cs).reshape(shape))
        if back:
            return {"psi": pos, "T": col}
        u0, u1, u2 = [t.double() for t in s["u0"]], [], []
        for a in range(3):
            v = torch.cat([_sample(u0, p, dx)[0] for p in pos[a].reshape(-1, 3).split(1 << 20)])
            t = (v * col[a].reshape(-1, 3)).sum(-1).reshape(u0[a].shape)
            nb = torch.stack([_shift(u0[a], d, st) for d in range(3) for st in (-1, 1)])
            u1.append(t)
            u2.append(torch.minimum(torch.maximum(t, nb.amin(0)), nb.amax(0)))
        c = sum(pos[a].narrow(a, 0, res[a]) + pos[a].narrow(a, 1, res[a]) for a in range(3)) / 6
        d0 = s["dye0"].double()
        dye = 0.5 * (_trilinear(d0, c.reshape(-1, 3), dx).reshape(d0.shape) - d0)
        return {"phi": pos, "F": col, "u1": u1, "u2": u2, "dye": dye}
    if kind == "project":
        return _project64([t.double() for t in s["u0"]], res)
    return _particles64(s, case, res, dx, dt)
