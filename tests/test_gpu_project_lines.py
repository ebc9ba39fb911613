"""The first and the last kernel of a projection around a solid, for both numbers
of cells of a line that a thread takes, against torch on the solver's own
divergence and pressure; and which grids the larger number meets."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def fields(res, seed):
    from edgeb200.fields import zeros_faces
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = zeros_faces(res)
    for t in u:
        t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
    return u


# a thread takes four cells of a line from 2^20 cells on, where a grid whose
# coarsest level fits has three levels or more, so that four divides its lines
@pytest.mark.gpu
@pytest.mark.parametrize("res", [(130, 64, 128), (131, 64, 128), (133, 64, 128)])
def test_lines_of_four_have_no_rest(res):
    from edgeb200 import EdgeError
    from edgeb200.projection import Projection
    for base_level in range(7):
        with pytest.raises(EdgeError):
            Projection(res, base_level=base_level)


# a box in the flow that begins and ends within groups, for lines of four and of
# two, which do and do not divide the axis
@pytest.mark.gpu
@pytest.mark.parametrize("res,base_level", [((136, 64, 128), 3), ((34, 32, 32), 4), ((19, 24, 32), 4)])
@pytest.mark.parametrize("inflow", [-0.5, 0.5])
def test_solid(res, base_level, inflow):
    from edgeb200.projection import Projection
    u = fields(res, 5)
    mask = torch.zeros(res, dtype=torch.int32, device="cuda")
    mask[res[0] - 7:res[0] - 1, 9:15, 10:23] = 1
    bvel = torch.zeros(res + (3,), device="cuda")
    bvel[..., 0], bvel[..., 1], bvel[..., 2] = 0.3, -0.2, 0.1
    for a in range(3):
        for side in range(2):
            u[a].select(a, side * res[a]).zero_()
    u[0][0] = inflow  # the one open side: its flux is the fluid's divergence
    before = [t.clone() for t in u]
    solid = mask > 0
    for a in range(3):  # the faces of solid cells carry the solid's velocity
        for side in range(2):
            part = before[a].narrow(a, side, res[a])
            part.copy_(torch.where(solid, bvel[..., a], part))
    P = Projection(res, base_level=base_level, boundary_types=((1, 2), (2, 2), (2, 2)), mask=mask, bvel=bvel)
    P.poisson(*u, max_iters=2)
    d = torch.zeros(res, device="cuda")
    for a in range(3):
        d = d + before[a].narrow(a, 1, res[a]) - before[a].narrow(a, 0, res[a])
    d = torch.where(solid, torch.zeros_like(d), d)
    fluid = ~solid
    # a fluid sum above zero has its mean taken off: a rounding of it and of the difference
    mean = float(d.double()[fluid].mean())
    assert abs(mean) > 1e-6  # far from zero, so that the sum's sign is not a matter of rounding
    want = torch.where(fluid, d.double() - max(mean, 0.0), 0.0)
    eps = np.finfo(np.float32).eps
    assert float((P.get("div").double() - want).abs().max()) <= 2 * eps * float(d.abs().max())
    x = P.get("p")
    assert float(x.abs().max()) > 0
    for a in range(3):
        xp = torch.nn.functional.pad(x, [0, 0] * (2 - a) + [1, 1])
        want = before[a] - (xp.narrow(a, 1, res[a] + 1) - xp.narrow(a, 0, res[a] + 1))
        for side in range(2):
            if (a, side) != (0, 0):
                want.select(a, side * res[a]).zero_()
        for side in range(2):
            part = want.narrow(a, side, res[a])
            part.copy_(torch.where(solid, bvel[..., a], part))
        assert torch.equal(u[a], want)
    P.close()
