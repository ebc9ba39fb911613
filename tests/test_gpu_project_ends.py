"""The first and the last kernel of a projection (divergence and initial
residual; gradient update), where a thread takes several cells of a line,
against torch on the solver's own divergence and pressure."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# lines of two cells, which do not divide every axis, and lines of four; walls and
# open sides; with and without a force buffer
@pytest.mark.gpu
@pytest.mark.parametrize("res,base_level", [((5, 6, 7), 2), ((17, 16, 24), 4), ((66, 32, 48), 4), ((128, 64, 136), 3)])
@pytest.mark.parametrize("bt,buffer", [(((2, 2), (2, 2), (2, 2)), True), (((2, 1), (1, 2), (1, 1)), False)])
def test_first_and_last_kernel(res, base_level, bt, buffer):
    from edgeb200.fields import zeros_faces
    from edgeb200.projection import Projection
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    u = zeros_faces(res)
    for t in u:
        t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
    for a in range(3):  # the walls' faces, as the solver sets them
        for side in range(2):
            if bt[a][side] == 2:
                u[a].select(a, side * res[a]).zero_()
    before = [t.clone() for t in u]
    f = zeros_faces(res) if buffer else None
    P = Projection(res, base_level=base_level, boundary_types=bt)
    P.poisson(*u, f=f, max_iters=2)
    d = torch.zeros(res, device="cuda")
    for a in range(3):  # the same additions in the same order
        d = d + before[a].narrow(a, 1, res[a]) - before[a].narrow(a, 0, res[a])
    assert torch.equal(P.get("div"), d)
    x = P.get("p")
    assert float(x.abs().max()) > 0
    for a in range(3):
        pad = [0, 0] * (2 - a) + [1, 1]
        xp = torch.nn.functional.pad(x, pad)
        grad = xp.narrow(a, 1, res[a] + 1) - xp.narrow(a, 0, res[a] + 1)
        want = before[a] - grad
        for side in range(2):
            if bt[a][side] == 2:
                want.select(a, side * res[a]).zero_()
        assert torch.equal(u[a], want)
        if buffer:
            assert torch.equal(f[a], -grad)
    P.close()
