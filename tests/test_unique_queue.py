"""The unique counter's device-built task queue: boards on both sides of its size rules, in an order that reuses and
grows the handle's buffers."""
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("boards", [(9, 10, 4, 11), (14, 13, 14, 5), (15, 16, 9, 15), (17, 18, 12, 17)])
def test_unique_queue_sizes(oracle_mod, boards):
    import nqueens
    eng = nqueens.Engine(0)
    try:
        for N in boards:
            r = eng.count_unique(N)
            assert (r.unique, r.total) == (oracle_mod.EXPECTED_UNIQUE[N], oracle_mod.EXPECTED_TOTAL[N]), N
    finally:
        eng.close()


@pytest.mark.parametrize("N", range(4, 17))
def test_unique_every_kind_of_board(oracle_mod, N):
    """Each size alone, on a handle of its own: boards that equal a rotation (x2, x4), boards with a rotation of the
    same first row, and part 1's (x8) all have to be told apart by the warp, for widths around half a warp too."""
    import nqueens
    eng = nqueens.Engine(0)
    try:
        r = eng.count_unique(N)
        assert (r.unique, r.total) == (oracle_mod.EXPECTED_UNIQUE[N], oracle_mod.EXPECTED_TOTAL[N])
    finally:
        eng.close()
