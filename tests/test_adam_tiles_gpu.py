"""GPU edge cases of the Adam step's SH tiles, whose number of Gaussians depends on the SH count: one less
than a tile, a whole one, one more, and several with a partial last one.  Oracle and tolerance as in
test_adam_edges_gpu."""
import pytest

from test_adam_edges_gpu import test_adam_step_edges as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,tile", [(1, 512), (2, 256), (3, 168), (4, 128), (5, 100), (9, 56), (13, 36), (15, 32), (16, 32)])
@pytest.mark.parametrize("tiles,more", [(1, -1), (1, 0), (1, 1), (3, 2)])
def test_adam_tiles(cuda, M, tile, tiles, more):
    check(cuda, tiles * tile + more, M, bf16=M % 2 == 1, aligned=True)
