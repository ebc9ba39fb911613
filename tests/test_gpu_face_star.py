"""The seven-point face stencils (velocity clamp, viscous force), where a thread
takes several faces along x, against torch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# one face a thread, two, and eight with axes that eight does not divide
@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((4, 4, 4), 0.25), ((5, 33, 9), 0.1), ((61, 64, 53), 1 / 64), ((99, 97, 101), 0.3),
                                    ((160, 64, 128), 1 / 64)])
def test_face_stencils(res, dx):
    from edgeb200 import ops
    from edgeb200.fields import zeros_faces
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    u, u1, got, vis = (zeros_faces(res) for _ in range(4))
    for t in u + u1:
        t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
    for t in got + vis:
        t.fill_(float("nan"))
    ops.clamp_u(u, u1, got)
    ops.lp_viscous(u1, dx, 5.5, vis)
    for a in range(3):
        near = []
        for d in range(3):
            n = u1[a].shape[d]
            i = torch.arange(n, device="cuda")
            near += [u1[a].index_select(d, (i + s).clamp(0, n - 1)) for s in (-1, 1)]
        near = torch.stack(near)
        assert torch.equal(got[a], u[a].clamp(near.amin(0), near.amax(0)))
        want = (near.double().sum(0) - 6 * u1[a].double()) / 5.5 / dx / dx
        # seven additions of terms up to six times the largest, three products
        tol = 10 * np.finfo(np.float32).eps * 12 * float(u1[a].abs().max()) / 5.5 / dx / dx
        assert float((vis[a].double() - want).abs().max()) <= tol
