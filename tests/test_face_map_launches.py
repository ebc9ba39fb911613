"""The launch count of the packed face map follows the library's rule, which sees
the spacing in float32 (no GPU)."""
import pytest

torch = pytest.importorskip("torch")


# a power of two; one in float32 only; none; axes whose clamp bound is no whole
# number in float32
@pytest.mark.parametrize("res,dx,want", [((66, 66, 66), 0.125, 1), ((66, 66, 66), 0.125 * (1 + 1e-9), 1),
                                         ((66, 66, 66), 0.125 * (1 + 1e-6), 2), ((66, 66, 34), 0.125, 2),
                                         ((66, 66, 35), 0.125, 1),
                                         ((4, 128, 128), 0.125, 2), ((128, 256, 66), 1 / 3, 2)])
def test_launches_of_the_packed_face_map(res, dx, want, monkeypatch):
    from edgeb200 import ops
    monkeypatch.setattr(ops.N, "call", lambda *a: None)
    monkeypatch.setattr(ops, "ptr", lambda *a: None)
    monkeypatch.setattr(ops, "stream", lambda *a: None)
    before = ops._launched[0]
    ops.face_map_packed(1, dx, None, res, [None] * 3, [None] * 3)
    assert ops._launched[0] - before == want
