"""Device memory of completion queries: sized to the query, and a level less where the device has no room."""
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

MIB = 1 << 20


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("N,queens,most", [
    (8, [(0, 0)], 8), (12, [(0, 3), (7, 9)], 8), (14, [(2, 5)], 16), (17, [(3, 4), (9, 12)], 40),
    (20, [(2, 2), (10, 7)], 192), (22, [(0, 3), (8, 12), (15, 6), (20, 1)], 192)])
def test_a_query_takes_what_its_size_needs(N, queens, most):
    import nqueens
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    warm = nqueens.Engine(0, auto_tune=False)                   # loads the kernels
    want = warm.count_completions(N, queens)
    warm.close()
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        before = _free(torch)
        assert eng.count_completions(N, queens) == want
        held = before - _free(torch)
        assert held <= most * MIB, held
        assert eng.count_completions(N, queens) == want
        assert before - _free(torch) == held                    # and no more for the next one
    finally:
        eng.close()
    assert _free(torch) >= before


def test_a_device_with_little_room_left(oracle_mod):
    """Beside a reservation of nearly all of the device's memory a query of 18 rows runs with a level less."""
    import nqueens
    torch = pytest.importorskip("torch")
    N, queens = 20, [(2, 2), (10, 7)]
    eng = nqueens.Engine(0, auto_tune=False)
    want = eng.count_completions(N, queens)
    eng.close()
    eng = nqueens.Engine(0, auto_tune=False)
    hog = None
    try:
        assert eng.count_completions(8, []) == 92
        torch.cuda.empty_cache()
        hog = torch.empty(_free(torch) - 96 * MIB, dtype=torch.uint8, device="cuda")
        assert _free(torch) < 128 * MIB
        assert eng.count_completions(N, queens) == want
        assert eng.count_completions(14, []) == oracle_mod.EXPECTED_TOTAL[14]
        del hog
        torch.cuda.empty_cache()
        assert eng.count_completions(N, queens) == want
    finally:
        eng.close()
        torch.cuda.empty_cache()
