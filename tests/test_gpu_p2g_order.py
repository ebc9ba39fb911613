"""The particle-to-grid scatter of ops.lp_p2g above the size at which it groups
the particles by cell: orders for which the library groups and orders for which
it scatters directly, and without the workspace, against the same sums in
float64."""
import numpy as np
import pytest

from test_gpu_p2g_grouped import scatter

torch = pytest.importorskip("torch")


def positions(order, res, num, rng):
    if order == "lattice":  # consecutive particles a cell and a bit apart
        k = np.arange(num)
        line = int((res[2] - 7) / 1.1)
        p = np.stack([3.3 + (k // line // 40) % (res[0] - 7), 3.4 + (k // line) % (res[1] - 7), 3.2 + 1.1 * (k % line)], 1)
    elif order == "outside":
        p = rng.random((num, 3)) * 2.9
    else:
        p = rng.random((num, 3)) * np.array(res)
        if order == "sorted":
            c = p.astype(np.int64)
            p = p[np.argsort((c[:, 0] * 64 + c[:, 1]) * 64 + c[:, 2], kind="stable")]
        elif order == "half":  # random ones and a lattice
            p[:num // 2] = positions("lattice", res, num // 2, rng)
    return p.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["lattice", "outside", "random", "sorted", "half"])
@pytest.mark.parametrize("workspace", [True, False])
def test_scatter_of_an_order(order, workspace, monkeypatch):
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    res, num = (20, 48, 40), 40000
    rng = np.random.default_rng(4)
    L = [float(n) for n in res]
    pos = positions(order, res, num, rng)
    val = rng.standard_normal((num, 3)).astype(np.float32)
    rad = (0.005 + 0.005 * rng.random(num)).astype(np.float32)
    ref, size, count = scatter(res, 1.0, val, pos, rad, 0.01, np.array(L))
    cu = lambda a: torch.as_tensor(a, device="cuda").contiguous()  # noqa: E731
    drag = zeros_faces(res)
    for t in drag:
        t.fill_(7.0)  # the call zeroes the fields
    if not workspace:  # no room for it: torch's allocator raises
        def full(*args, **kw):
            raise torch.cuda.OutOfMemoryError("full")
        monkeypatch.setattr(torch, "empty", full)
    v, p, r = cu(val), cu(pos), cu(rad)
    before = ops.launch_count()
    ops.lp_p2g(res, 1.0, drag, v, p, r, num, 0.01, L)
    assert ops.launch_count() - before == (5 if workspace else 1)
    monkeypatch.undo()
    # a term has a dozen roundings (the weights' from coordinates of up to 48
    # cells: 48 eps each in three factors), the sum one per particle
    eps = np.finfo(np.float32).eps
    for a in range(3):
        err = np.abs(drag[a].cpu().numpy().astype(np.float64) - ref[a])
        lim = eps * ((count + 12) * size[a] + 3 * 48 * max(1.0, float(np.abs(val).max())) * count)
        assert np.all(err <= lim), float((err - lim).max())
