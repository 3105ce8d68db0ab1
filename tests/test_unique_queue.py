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
