"""Record lists beside a reservation of nearly all of the device's memory: a queue whose bound has no room is built at
its length."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

MIB = 1 << 20


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("m", [16384, 16385])          # short: bound of 52 MiB; long: guess of 17 MiB; 10 MiB needed
def test_a_device_with_little_room_left(m):
    import nqueens
    torch = pytest.importorskip("torch")
    N = 17
    r = np.ascontiguousarray(nqueens.gen_records(N)[:m])
    eng = nqueens.Engine(0, auto_tune=False)
    want = eng.exec_records(N, r, want_solutions=True)
    items = eng.last_run_info()[1]
    eng.close()
    assert 16 * items < 12 * MIB
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        eng.exec_records(N, r[:100], want_solutions=True)
        torch.cuda.empty_cache()
        hog = torch.empty(_free(torch) - 20 * MIB, dtype=torch.uint8, device="cuda")
        assert _free(torch) < 24 * MIB
        for _ in range(2):
            got = eng.exec_records(N, r, want_solutions=True)
            assert got[0] == want[0] and np.array_equal(got[1], want[1])
            assert eng.last_run_info()[1] == items
        del hog
    finally:
        eng.close()
        torch.cuda.empty_cache()
