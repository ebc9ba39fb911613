"""What the marches of fields check and allocate on the host, before anything
is launched (no GPU)."""
import pytest

torch = pytest.importorskip("torch")


def _fields(res, count):
    return [torch.zeros(res + (3,)) for _ in range(count)]


# the results are written into the accumulated map by the dimensions of the new
# one: a map of another size has to be refused, as a copy refuses it
@pytest.mark.parametrize("at", range(7))
@pytest.mark.parametrize("other", [(8, 8, 6), (8, 8, 12)])
def test_accumulated_map_of_another_size_is_refused(at, other):
    from sim import hermite
    res, dx = (8, 8, 8), 0.125
    u = [torch.zeros(s) for s in ((9, 8, 8), (8, 9, 8), (8, 8, 9))]
    acc = _fields(res, 7)
    acc[at] = _fields(other, 1)[0]
    with pytest.raises(ValueError, match="size mismatch"):
        hermite.advect_psi_garm_ed4_fusion_unroll(*_fields(res, 7), *acc, *u, None, dx, 0.01, 0.01)
    if at < 4:
        with pytest.raises(ValueError, match="size mismatch"):
            hermite.advect_ps_hermite_ed4_fd_unroll(*_fields(res, 4), *acc[:4], *u, None, dx, 0.01, 0.01)


# the packed copy of the map is float32 whatever torch's default type is
@pytest.mark.parametrize("dtype", [torch.float64, torch.float16, torch.bfloat16, torch.float32])
def test_scratch_under_another_default_dtype(dtype, monkeypatch):
    from edgeb200 import ops
    res = (4, 5, 6)
    u = [torch.zeros(s) for s in ((5, 5, 6), (4, 6, 6), (4, 5, 7))]
    m, o = _fields(res, 7), _fields(res, 7)
    seen, empty = [], torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: seen.append(empty(*a, **k)) or seen[-1])
    before = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        with pytest.raises(ValueError, match="CUDA"):  # tensors of the host go no further
            ops.march_edge(u, 0.25, 0.01, 0.01, m[0], m[1:4], m[4:], o[0], o[1:4], o[4:])
        with pytest.raises(ValueError, match="CUDA"):
            ops.march_ed4(u, 0.25, 0.01, 0.01, m[0], m[1:4], o[0], o[1:4])
    finally:
        torch.set_default_dtype(before)
    assert [(t.dtype, t.numel()) for t in seen] == [(torch.float32, 8 * 4 * 4 * 5 * 6)] * 2
