"""Marches and semi-Lagrangian advection by tiles of cells, whose velocity
samples come from shared memory (or, from a warp with a sample outside the
tile, from global memory): the marches, of packed maps and of fields through a
packed copy, against the ones straight from the fields, which always read
global memory, the advection against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# one tile; tiles filled exactly; ragged tiles that both rules, one and none
# accept; a flow that stays in the tile and one that leaves it
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((4, 4, 8), 1 / 8), ((12, 8, 16), 1 / 8), ((39, 40, 56), 1 / 40),
                                    ((15, 16, 24), 1 / 16), ((16, 15, 23), 1 / 23), ((9, 17, 33), 1 / 32)])
@pytest.mark.parametrize("cells", [0.3, 3.0])
@pytest.mark.parametrize("variant", [0, 1, 2, "identity"])
def test_march_by_tiles(res, dx, cells, variant, monkeypatch):
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    identity, variant = variant == "identity", 1 if variant == "identity" else variant
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    rnd = lambda *s: 2 * torch.rand(*s, generator=g, device="cuda") - 1  # noqa: E731
    u = zeros_faces(res)
    for t in u:
        t.copy_(rnd(*t.shape))
    dt, eps = cells * dx, 0.125 * dx  # speeds up to one
    X = torch.stack(torch.meshgrid(*[(torch.arange(n, device="cuda") + 0.5) * dx for n in res], indexing="ij"), -1)
    psi = X.contiguous() if identity else (X + 0.3 * dx * rnd(*res, 3)).contiguous()
    T = [((0.0 if identity else 0.1) * rnd(*res, 3) + torch.eye(3, device="cuda")[c]).contiguous() for c in range(3)]
    dT = [torch.zeros(*res, 3, device="cuda") if identity else rnd(*res, 3) for _ in range(3)] if variant else None
    d2T = [rnd(*res) for _ in range(3)] if variant == 2 else None
    vec = lambda: torch.empty(*res, 3, device="cuda")  # noqa: E731
    o = [vec() for _ in range(7)] + [torch.empty(res, device="cuda") for _ in range(3)]
    q = [vec() for _ in range(7)] + [torch.empty(res, device="cuda") for _ in range(3)]
    packed = torch.zeros((ops.PLANES[variant],) + res + (4,), device="cuda")
    out = torch.full_like(packed, float("nan"))
    ops.map_pack(variant, psi, T, dT, d2T, packed)
    ops.march_packed(variant, u, dx, dt, eps, packed, out, res, identity=identity)
    f = [vec() for _ in range(7)]
    state = [t.clone() for t in [psi, *T, *(dT or [])]]
    if variant == 1:
        ops.march_edge(u, dx, dt, eps, state[0], state[1:4], state[4:7], f[0], f[1:4], f[4:7], identity=identity,
                       update=True)
    elif variant == 0:
        ops.march_ed4(u, dx, dt, eps, state[0], state[1:4], f[0], f[1:4], update=True)
    # straight from the fields; the identity map as any other
    monkeypatch.setattr(ops, "_map_workspace", lambda psi: None)
    if variant == 1:
        ops.march_edge(u, dx, dt, eps, psi, T, dT, o[0], o[1:4], o[4:7])
    elif variant == 0:
        ops.march_ed4(u, dx, dt, eps, psi, T, o[0], o[1:4])
    else:
        ops.march_ed8(u, dx, dt, eps, psi, T, dT, d2T, o[0], o[1:4], o[4:7], o[7:10])
    ops.map_unpack(variant, out, q[0], q[1:4], q[4:7] if variant else None, q[7:10] if variant == 2 else None)
    # a marched position: a rounding or two of its own, times the flow's
    # stretching in one step (RK4 of a velocity that changes by two per cell);
    # the map's slope is below four, its curvature below eight over dx
    ulp = np.finfo(np.float32).eps * (float(psi.abs().max()) + dx)
    s = 2 * cells
    tol = 4 * ulp * 2 * (1 + s + s**2 / 2 + s**3 / 4 + s**4 / 24)
    tol_T = tol / eps if variant != 1 else 8 * tol / dx
    for r in [q] if variant == 2 else [q, f]:
        assert float((r[0] - o[0]).abs().max()) <= 4 * tol
        for a, b in zip(r[1:4], o[1:4]):
            assert float((a - b).abs().max()) <= tol_T * (1 + s)**3
        for a, b in zip(r[4:7], o[4:7]):
            if variant:
                assert float((a - b).abs().max()) <= tol_T * (1 + s)**3 / eps
    if variant != 2:
        assert all(torch.equal(a, b) for a, b in zip(state, f))


# the smallest grids that take tiles, a ragged one and one just below
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((72, 72, 72), 1 / 64), ((75, 72, 71), 1 / 72), ((88, 64, 64), 1 / 64),
                                    ((70, 70, 70), 1 / 70)])
@pytest.mark.parametrize("cells", [0.3, 3.0])
def test_advect_by_tiles(res, dx, cells):
    from edgeb200 import ops
    from oracle import edge_oracle as O
    rng = np.random.default_rng(5)
    u = [rng.uniform(-1, 1, size=s).astype(np.float32) for s in O.face_shapes(res)]
    dt = np.float32(cells * dx)
    want = O.advect_u_semi_lagrangian(u, dx, dt)
    got = [torch.full(s, float("nan"), device="cuda") for s in O.face_shapes(res)]
    ops.advect_u_sl([torch.from_numpy(t).cuda() for t in u], dx, float(dt), got)
    # two roundings of the position, times the flow's stretching in one step,
    # times the velocity's change of two per cell
    s = 2 * cells
    tol = 8 * np.finfo(np.float32).eps * max(res) * 2 * (1 + s + s**2 / 2 + s**3 / 4 + s**4 / 24)
    for a, b in zip(got, want):
        assert np.abs(a.cpu().numpy() - b).max() <= tol
