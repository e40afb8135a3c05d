"""The state buffers' size queries never shrink as a scene or batch grows: a buffer sized for the largest
scene a program will hold is accepted for every smaller one (after pruning, say).  No GPU."""
import pytest

from omnigs_b200 import capi


def _never_shrinks(sizes):
    return all(b >= a for a, b in zip(sizes, sizes[1:]))


def test_geometry_bytes_never_shrink():
    # the depth sort's tiles change size with P: every step of 64, and single steps around the changes
    steps = sorted(set(range(0, 400000, 64)) | {p + d for p in range(0, 400000, 1024) for d in (-1, 0, 1) if p + d >= 0})
    assert _never_shrinks([capi.geom_bytes(p) for p in steps])


@pytest.mark.parametrize("V", [1, 2, 3, 7, 16, 32])
def test_batch_state_bytes_never_shrink(V):
    sizes = [(512, 256)] * V
    steps = sorted({p + d for p in range(0, 170000, 512) for d in (-1, 0, 1) if p + d >= 0})
    assert _never_shrinks([capi.batch_state_bytes(p, sizes) for p in steps])


@pytest.mark.parametrize("P", [500, 5000, 12289, 20480, 81920, 163840])
def test_batch_state_bytes_never_shrink_with_views(P):
    assert _never_shrinks([capi.batch_state_bytes(P, [(512, 256)] * v) for v in range(1, 33)])
