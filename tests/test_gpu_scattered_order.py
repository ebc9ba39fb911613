"""Velocity samples at points: a warp takes a row's taps by wide or by single
loads, whichever the order of its points favours.  The order must not change a
point's value."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# orders that take single loads, wide ones and both by turns; a last warp that
# is not full; points in the first and last rows, where wide loads would pass
# the ends of the fields, and beyond the box
@pytest.mark.gpu
@pytest.mark.parametrize("res", [(4, 4, 4), (9, 7, 11), (24, 20, 33)])
@pytest.mark.parametrize("num", [1, 31, 33, 5000])
def test_order_of_points(res, num):
    from edgeb200 import ops
    rng = np.random.default_rng(8)
    shapes = [[n + (d == a) for d, n in enumerate(res)] for a in range(3)]
    u = [torch.from_numpy(rng.uniform(-1, 1, size=s).astype(np.float32)).cuda() for s in shapes]
    pts = (rng.uniform(-1, 1, size=(num, 3)) * (np.array(res) + 2) / 2 + np.array(res) / 2).astype(np.float32)
    cell = np.clip(pts, 0, None).astype(np.int64)
    key = (cell[:, 0] * 64 + cell[:, 1]) * 64 + cell[:, 2]
    by_cell = np.argsort(key, kind="stable")
    runs = by_cell.reshape(-1, 4)[rng.permutation(num // 4)].reshape(-1) if num % 4 == 0 else by_cell[::-1]
    half = np.concatenate([by_cell[:num // 2], rng.permutation(by_cell[num // 2:])])
    vel = torch.zeros((num, 3), device="cuda")
    out = []
    for order in (np.arange(num), by_cell, runs, half):
        pos = torch.from_numpy(np.ascontiguousarray(pts[order])).cuda()
        acc, vd = torch.full_like(vel, float("nan")), torch.full_like(vel, float("nan"))
        ops.lp_acc(u, 1.0, vel, pos, acc, num, 0.0, 1.0, 0.0)
        ops.lp_vel_diff(u, 1.0, vel, vd, pos, num, 0.066, 2 / 3, 35.0)
        v = ops.points_mac(u, 1.0, pos)[0]
        back = torch.from_numpy(np.argsort(order)).cuda()
        out.append([t[back] for t in (acc, vd, v)])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert torch.equal(a, b)
    assert torch.equal(out[0][0], out[0][2])  # at rest and without drag the acceleration is the sample
