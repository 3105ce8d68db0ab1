"""The fused prepare + split launch: its queue's capacity rules give the same per-record counts on every side of them."""
import ctypes

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.fixture(scope="module")
def eng():
    import nqueens
    e = nqueens.Engine(0, auto_tune=False)
    yield e
    e.close()


def _sample(N, m):
    import nqueens
    recs = nqueens.gen_records_starts(N, 0, 40) if N > 20 else nqueens.gen_records(N)
    at = np.sort(np.random.default_rng(N * 7 + m).choice(len(recs), m, replace=False))
    return np.ascontiguousarray(recs[at])


@pytest.mark.parametrize("N,m", [(13, 7), (15, 16384), (15, 16385), (17, 16385), (22, 300), (22, 17000)])
def test_every_depth_gives_the_same_counts(eng, N, m):
    """Lists on both sides of the read-back limit, and large boards, where 8 items a level are too few: every
    split depth gives the unsplit counts."""
    recs = _sample(N, m)
    want = None
    for split in (0, 1, 2, 3, -1):
        if N == 22 and m > 1000 and split in (0, 3):
            continue
        eng.set_config(64, 0, split)
        total, sol = eng.exec_records(N, recs, want_solutions=True)
        want = sol if want is None else want
        assert np.array_equal(sol, want), split
        assert total == int(want.sum())
    eng.set_config(64, 0, -1)


@pytest.mark.parametrize("N,m", [(14, 1), (16, 20011), (17, 49207), (22, 30001), (22, 57000)])
def test_noalloc_queue_in_the_fixed_scratch(eng, N, m):
    """The no-allocation call splits as far as its scratch holds the queue: per record the regular call's counts."""
    _check_noalloc(eng, N, _sample(N, m))


@pytest.mark.parametrize("m", [20000, 21700, 24000])
def test_noalloc_queue_longer_than_expected(eng, m):
    """The eighth of N=17's list with the most frames a task, over and over: two levels make 42 items a task where
    41 are expected.  The queue fits (20,000), does not though it should (21,700: built again), or should not."""
    import nqueens
    recs = nqueens.gen_records(17)
    recs = np.ascontiguousarray(np.resize(recs[:len(recs) // 8], m))
    _check_noalloc(eng, 17, recs)


def _check_noalloc(eng, N, recs):
    torch = pytest.importorskip("torch")
    import nqueens
    m = len(recs)
    want_total, want = eng.exec_records(N, recs, want_solutions=True)
    d_rec = torch.from_numpy(recs.view(np.uint8).copy()).cuda()
    d_total = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    d_sol = torch.full((m,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    st = nqueens.lib().nq_exec_solutions_noalloc(N, ctypes.c_void_p(d_rec.data_ptr()), m,
                                                 int((recs["startijkl"] >> 20).min()),
                                                 ctypes.c_void_p(d_sol.data_ptr()), ctypes.c_void_p(d_total.data_ptr()), None)
    assert st == 0 and int(d_total.item()) == want_total
    assert np.array_equal(d_sol.cpu().numpy().view(np.uint64), want)
