"""The particle-to-grid scatter through particles grouped by cell, against the
same sums in float64."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def n2(x):
    a = np.abs(x)
    return np.where(a < 0.5, 0.75 - a * a, np.where(a < 1.5, 0.5 * (1.5 - a) ** 2, 0.0))


def scatter(res, dx, vdiff, pos, rad, lrad, L):
    """lp.py:100-156 in float64: the drag, and the sums of its terms' sizes."""
    out, size, count = [], [], 0
    g = pos.astype(np.float32) / np.float32(dx)
    keep = np.all((pos >= np.float32(3 * dx)) & (pos <= np.float32(L) - np.float32(3 * dx)), axis=1)
    g, v = g[keep].astype(np.float64), vdiff[keep].astype(np.float64)
    s = (rad[keep].astype(np.float64) / lrad) ** 3
    for a in range(3):
        dim = [n + (d == a) for d, n in enumerate(res)]
        f, m, c = np.zeros(dim), np.zeros(dim), np.zeros(dim)
        q = [g[:, d] - (0.0 if d == a else 0.5) for d in range(3)]
        b = [np.floor(x).astype(int) - 1 for x in q]
        for o in np.ndindex(4, 4, 4):
            ix = [b[d] + o[d] for d in range(3)]
            w = n2(q[0] - ix[0]) * n2(q[1] - ix[1]) * n2(q[2] - ix[2])
            ok = np.all([(ix[d] >= 0) & (ix[d] < dim[d]) for d in range(3)], axis=0) & (w != 0)
            at = tuple(x[ok] for x in ix)
            np.add.at(f, at, (v[:, a] * w * s)[ok])
            np.add.at(m, at, np.abs(v[:, a] * w * s)[ok])
            np.add.at(c, at, 1.0)
        out.append(f)
        size.append(m)
        count = max(count, int(c.max(initial=0)))
    return out, size, count


# one particle, a warp's edges, a batch's edges, several batches per warp
# (more than 32 warps per SM), all in one cell, a domain larger than the grid
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx,num,spread,over", [
    ((12, 10, 9), 1.0, 1, 1.0, 0.0), ((12, 10, 9), 1.0, 31, 1.0, 0.0), ((12, 10, 9), 0.5, 33, 0.02, 0.0),
    ((16, 33, 20), 1 / 20, 4097, 1.0, 0.0), ((8, 8, 8), 1.0, 700, 1.0, 6.0), ((40, 24, 32), 1 / 24, 330000, 1.0, 0.0)])
def test_grouped_scatter(res, dx, num, spread, over):
    from edgeb200 import _native as N
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    rng = np.random.default_rng(3)
    L = np.array([n * dx + over * dx for n in res])
    pos = (rng.random((num, 3)) * L * spread + L * 0.5 * (1 - spread)).astype(np.float32)
    val = rng.standard_normal((num, 3)).astype(np.float32)
    rad = (0.005 + 0.005 * rng.random(num)).astype(np.float32)
    ref, size, count = scatter(res, dx, val, pos, rad, 0.01, L)
    cu = lambda a: torch.as_tensor(a, device="cuda").contiguous()  # noqa: E731
    p, v, r, drag = cu(pos), cu(val), cu(rad), zeros_faces(res)
    work = ops._p2g_workspace(res, num, p.device)
    args = lambda w: ["edge_lp_p2g_grouped", *res, ops.F(dx), *ops._p3(drag), ops.ptr(v), ops.ptr(p), ops.ptr(r), num,  # noqa: E731
                      ops.F(0.01), *[ops.F(x) for x in L], ctypes.c_void_p(w.data_ptr()), ctypes.c_longlong(w.numel()),
                      ops.stream()]
    for t in drag:
        t.fill_(7.0)  # the call zeroes the fields
    N.call(*args(work))
    # a term has a dozen roundings (the weights' from coordinates of up to 40
    # cells: 40 eps each in three factors), the sum one per particle
    eps = np.finfo(np.float32).eps
    for a in range(3):
        err = np.abs(drag[a].cpu().numpy().astype(np.float64) - ref[a])
        lim = eps * ((count + 12) * size[a] + 3 * 40 * max(1.0, float(np.abs(val).max())) * count)
        assert np.all(err <= lim), float((err - lim).max())
    with pytest.raises(N.EdgeError):
        N.call(*args(work[:-1]))


@pytest.mark.gpu
def test_not_finite_values_reach_only_their_faces():
    from edgeb200 import _native as N
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    res = (10, 10, 10)
    pos = torch.tensor([[4.2, 5.7, 5.1], [4.6, 5.3, 5.2], [float("nan"), 5.0, 5.0]], device="cuda")
    val = torch.tensor([[1.0, float("inf"), 2.0], [3.0, 1.0, float("nan")], [1.0, 1.0, 1.0]], device="cuda")
    rad = torch.full((3,), 0.01, device="cuda")
    got, want = zeros_faces(res), zeros_faces(res)
    tail = [ops.ptr(val), ops.ptr(pos), ops.ptr(rad), 3, ops.F(0.01), *[ops.F(10.0)] * 3]
    work = ops._p2g_workspace(res, 3, pos.device)
    N.call("edge_lp_p2g_grouped", *res, ops.F(1.0), *ops._p3(got), *tail, ctypes.c_void_p(work.data_ptr()),
           ctypes.c_longlong(work.numel()), ops.stream())
    N.call("edge_lp_p2g", *res, ops.F(1.0), *ops._p3(want), *tail, ops.stream())
    for a, b in zip(got, want):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
