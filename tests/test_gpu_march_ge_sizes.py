"""The packed GE march at the sizes where its form changes, against the march in
the reference's layout."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# the smallest grid, the largest that keeps its registers and the smallest that
# does not, for spacings that are and are not a power of two
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((4, 4, 4), 0.25), ((48, 32, 64), 1 / 32), ((49, 32, 64), 1 / 32),
                                    ((5, 9, 33), 1 / 9), ((64, 64, 64), 1 / 63), ((65, 64, 64), 1 / 63)])
@pytest.mark.parametrize("cells", [0.5, 3.0])
def test_ge_march_forms(res, dx, cells):
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    g = torch.Generator(device="cuda")
    g.manual_seed(13)
    rnd = lambda *s: 2 * torch.rand(*s, generator=g, device="cuda") - 1  # noqa: E731
    u = zeros_faces(res)
    for t in u:
        t.copy_(0.2 * rnd(*t.shape))
    X = torch.stack(torch.meshgrid(*[(torch.arange(n, device="cuda") + 0.5) * dx for n in res], indexing="ij"), -1)
    psi = (X + 0.3 * dx * rnd(*res, 3)).contiguous()
    T = [(0.1 * rnd(*res, 3) + torch.eye(3, device="cuda")[c]).contiguous() for c in range(3)]
    dT, d2T = [rnd(*res, 3) for _ in range(3)], [rnd(*res) for _ in range(3)]
    packed = torch.zeros((8,) + res + (4,), device="cuda")
    out = torch.full_like(packed, float("nan"))
    ops.map_pack(2, psi, T, dT, d2T, packed)
    ops.march_ge_packed(u, dx, cells * dx, packed, out, res)
    vec = lambda: torch.empty(*res, 3, device="cuda")  # noqa: E731
    o, q = [vec() for _ in range(7)], [vec() for _ in range(7)]
    o2, q2 = ([torch.empty(res, device="cuda") for _ in range(3)] for _ in range(2))
    ops.march_ge(u, dx, cells * dx, psi, T, dT, d2T, o[0], o[1:4], o[4:7], o2)
    ops.map_unpack(2, out, q[0], q[1:4], q[4:7], q2)
    # a marched position: a rounding or two of its own, times the flow's
    # stretching in one step (RK4 of a velocity that changes by 0.4 per cell);
    # the map's slope is below four, its curvature below eight over dx
    s = 0.4 * cells
    tol = 8 * np.finfo(np.float32).eps * (float(psi.abs().max()) + dx) * (1 + s + s**2 / 2 + s**3 / 4 + s**4 / 24)
    assert float((q[0] - o[0]).abs().max()) <= 4 * tol
    for a, b in zip(q[1:4], o[1:4]):
        assert float((a - b).abs().max()) <= 8 * tol / dx * (1 + s)**3
