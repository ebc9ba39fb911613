"""Marches by tiles of cells do the arithmetic of the marches by consecutive
cells: the same cells in a grid that takes tiles and in a larger one that does
not, and of fields through a packed copy, give the same bits."""
import pytest

torch = pytest.importorskip("torch")


def inputs(res, dx, seed):
    from edgeb200.fields import zeros_faces
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rnd = lambda *s: 2 * torch.rand(*s, generator=g, device="cuda") - 1  # noqa: E731
    u = zeros_faces(res)
    for t in u:
        t.copy_(rnd(*t.shape))  # speeds up to one
    X = torch.stack(torch.meshgrid(*[(torch.arange(n, device="cuda") + 0.5) * dx for n in res], indexing="ij"), -1)
    psi = (X + 0.3 * dx * rnd(*res, 3)).contiguous()
    T = [(0.1 * rnd(*res, 3) + torch.eye(3, device="cuda")[c]).contiguous() for c in range(3)]
    return u, psi, T, [rnd(*res, 3) for _ in range(3)], [rnd(*res) for _ in range(3)]


def march(variant, identity, u, dx, dt, psi, T, dT, d2T):
    from edgeb200 import ops
    res = tuple(psi.shape[:3])
    packed = torch.zeros((ops.PLANES[variant],) + res + (4,), device="cuda")
    out = torch.full_like(packed, float("nan"))
    ops.map_pack(variant, psi, T, dT if variant else None, d2T if variant == 2 else None, packed)
    ops.march_packed(variant, u, dx, dt, 0.125 * dx, packed, out, res, identity=identity)
    return out


# 24^3 fills its tiles, 25^3 fills six tenths of them; at 24x24x32 with a spacing
# that is a power of two the ED4 march takes no tiles, at 24x24x40 it does.  A
# flow that stays in the tiles and one that leaves them by two cells
@pytest.mark.gpu
@pytest.mark.parametrize("small,large,dx", [((24, 24, 24), (25, 25, 25), 1 / 32), ((24, 24, 24), (25, 25, 25), 1 / 24),
                                            ((24, 24, 32), (24, 24, 40), 1 / 32)])
@pytest.mark.parametrize("cells", [0.3, 3.0])
@pytest.mark.parametrize("variant", [0, 1, 2, "identity"])
def test_same_bits_with_and_without_tiles(small, large, dx, cells, variant):
    identity, variant = variant == "identity", 1 if variant == "identity" else variant
    u, psi, T, dT, d2T = inputs(large, dx, 17)
    cut = lambda t, a=None: t[tuple(slice(0, n + (d == a)) for d, n in enumerate(small))].contiguous()  # noqa: E731
    big = march(variant, identity, u, dx, cells * dx, psi, T, dT, d2T)
    less = march(variant, identity, [cut(t, a) for a, t in enumerate(u)], dx, cells * dx, cut(psi),
                 [cut(t) for t in T], [cut(t) for t in dT], [cut(t) for t in d2T])
    # three cells of flow and the stencils of samples, map and derived planes
    # away from the sides at which the grids differ
    at = (slice(None),) + tuple(slice(0, n - 10 if n != m else n) for n, m in zip(small, large)) + (slice(0, 3),)
    assert torch.isfinite(big[at]).all()
    assert torch.equal(big[at], less[at])


# in tiles and not, where a division by the spacing is exact and where it is not
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((24, 24, 24), 1 / 32), ((24, 24, 24), 1 / 24), ((25, 25, 25), 1 / 32),
                                    ((9, 17, 33), 1 / 17)])
@pytest.mark.parametrize("cells", [0.3, 3.0])
@pytest.mark.parametrize("variant", [0, 1])
def test_fields_through_a_packed_copy(res, dx, cells, variant, monkeypatch):
    from edgeb200 import ops
    u, psi, T, dT, _ = inputs(res, dx, 19)
    dt, eps = cells * dx, 0.125 * dx
    vec = lambda: torch.full((*res, 3), float("nan"), device="cuda")  # noqa: E731

    def fields():
        o = [vec() for _ in range(4 + 3 * variant)]
        if variant:
            ops.march_edge(u, dx, dt, eps, psi, T, dT, o[0], o[1:4], o[4:])
        else:
            ops.march_ed4(u, dx, dt, eps, psi, T, o[0], o[1:])
        return o

    got = fields()
    q = [vec() for _ in range(7)]
    ops.map_unpack(variant, march(variant, False, u, dx, dt, psi, T, dT, None), q[0], q[1:4],
                   q[4:] if variant else None, None)

    def full(*args, **kw):  # no room for the copy: torch's allocator raises
        raise torch.cuda.OutOfMemoryError("full")
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", full)
    straight = fields()
    monkeypatch.setattr(torch, "empty", empty)
    for a, b, c in zip(got, q, straight):
        assert torch.equal(a, b)
        assert torch.equal(a, c)
