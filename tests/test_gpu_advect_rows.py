"""Semi-Lagrangian advection of grids whose rows are whole 128-byte lines, which
takes tiles of cells from a larger size on than the others: against the
oracle on both sides of that size and below the others' one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("res,dx", [((72, 72, 64), 1 / 64), ((104, 104, 64), 1 / 104), ((106, 104, 64), 1 / 64),
                                    ((74, 100, 96), 1 / 96)])
@pytest.mark.parametrize("cells", [0.5, 3.0])
def test_advect_rows_of_whole_lines(res, dx, cells):
    from edgeb200 import ops
    from oracle import edge_oracle as O
    rng = np.random.default_rng(6)
    u = [rng.uniform(-1, 1, size=s).astype(np.float32) for s in O.face_shapes(res)]
    dt = np.float32(cells * dx)
    want = O.advect_u_semi_lagrangian(u, dx, dt)
    got = [torch.full(s, float("nan"), device="cuda") for s in O.face_shapes(res)]
    ops.advect_u_sl([torch.from_numpy(t).cuda() for t in u], dx, float(dt), got)
    # two roundings of the position, times the flow's stretching in one step,
    # times the velocity's change of two per cell
    s = 2 * cells
    tol = 8 * np.finfo(np.float32).eps * max(res) * 2 * (1 + s + s**2 / 2 + s**3 / 4 + s**4 / 24)
    for a, b in zip(got, want):
        assert np.abs(a.cpu().numpy() - b).max() <= tol
