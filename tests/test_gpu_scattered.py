"""Velocity samples at scattered points take a row's taps by wide loads: against
the sampler with gradient, which loads them one by one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# rows of every alignment (odd sizes, fields that start on any word), the
# corners, where a wide load would pass an end of the field, and beyond them
@pytest.mark.gpu
@pytest.mark.parametrize("res", [(4, 4, 4), (5, 7, 9), (8, 6, 11), (16, 12, 20)])
@pytest.mark.parametrize("word", [0, 1, 2, 3])
def test_scattered_samples(res, word):
    from edgeb200 import ops
    rng = np.random.default_rng(3)
    u = []
    for a in range(3):
        s = [n + (d == a) for d, n in enumerate(res)]
        buf = torch.full((int(np.prod(s)) + 8,), float("nan"), device="cuda")
        f = buf[word:word + int(np.prod(s))].view(*s)
        f.copy_(torch.from_numpy(rng.uniform(-1, 1, size=s)))
        u.append(f)
    lo, hi = -1.0, np.array(res) + 1.0
    pts = rng.uniform(0, 1, size=(5000, 3)) * (hi - lo) + lo
    pts[:8] = [[(lo, hi[d])[c >> d & 1] for d in range(3)] for c in range(8)]
    pos = torch.as_tensor(pts.astype(np.float32), device="cuda").contiguous()
    v, vg, _ = ops.points_mac(u, 1.0, pos)
    vel, vd = torch.zeros_like(pos), torch.empty_like(pos)
    ops.lp_vel_diff(u, 1.0, vel, vd, pos, 5000, 0.066, 2 / 3, 35.0)
    acc = torch.full_like(pos, float("nan"))
    ops.lp_acc(u, 1.0, vel, pos, acc, 5000, 0.0, 1.0, 0.0)
    # both sum the same 27 products of values up to one with weights that sum
    # to one: a rounding per multiply-add of the three levels, two per weight
    tol = 16 * np.finfo(np.float32).eps
    assert float((v - vg).abs().max()) <= tol
    assert float((acc - vg).abs().max()) <= tol
    k = -float((vd * vg).sum() / (vg * vg).sum())  # the drag's factor
    assert k > 0 and float((vd + k * vg).abs().max()) <= 2 * tol * k
