"""The packed face map takes a face's psi and Jacobian column from the two
cells it separates where the full Hermite contraction's other terms vanish,
and from the full contraction elsewhere: both against the reference-layout
face map, which always contracts all 64 coefficients."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# the smallest grid; short axes, whose clamp bound lies below the last cell;
# long power-of-two axes, where every face is on a line; spacings that are no
# power of two, with a block's worth of faces and more
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((4, 4, 4), 0.25), ((5, 7, 33), 1 / 32), ((64, 64, 65), 1 / 64),
                                    ((66, 64, 130), 1 / 64), ((24, 40, 56), 1 / 40), ((61, 75, 9), 1 / 75)])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_face_map_on_lines_and_off(res, dx, variant):
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    X = torch.stack(torch.meshgrid(*[(torch.arange(n, device="cuda") + 0.5) * dx for n in res], indexing="ij"), -1)
    psi = (X + 0.3 * dx * rnd(*res, 3)).contiguous()
    T = [(0.1 * rnd(*res, 3) + torch.eye(3, device="cuda")[c]).contiguous() for c in range(3)]
    dT = [rnd(*res, 3) for _ in range(3)] if variant else None
    d2T = [rnd(*res) for _ in range(3)] if variant == 2 else None
    packed = torch.zeros((ops.PLANES[variant],) + res + (4,), device="cuda")
    ops.map_pack(variant, psi, T, dT, d2T, packed)
    fp, fc, rp, rc = (zeros_faces(res, 3) for _ in range(4))
    for t in fp + fc:
        t.fill_(float("nan"))  # every face is written
    ops.face_map_packed(variant, dx, packed, res, fp, fc)
    ops.face_map(variant, dx, psi, T, dT, d2T, rp, rc)
    # a value is a sum of products of O(psi); a column is such a sum, with
    # coefficients up to 1.5, divided by dx: four roundings of each
    eps, top = np.finfo(np.float32).eps, float(psi.abs().max()) + dx * 8
    for a in range(3):
        assert float((fp[a] - rp[a]).abs().max()) <= 4 * eps * top
        assert float((fc[a] - rc[a]).abs().max()) <= 4 * eps * 1.5 * top / dx
