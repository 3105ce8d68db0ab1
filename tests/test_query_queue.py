"""Completion queries from the device-built queue: boards on both sides of its level rules, and queens on neighbouring
rows (multi-row steps, wide schedule words)."""
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.fixture(scope="module")
def eng():
    import nqueens
    e = nqueens.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7, 11, 12, 13, 14, 15, 16, 18])
def test_empty_board(eng, oracle_mod, N):
    assert eng.count_completions(N, []) == oracle_mod.EXPECTED_TOTAL[N]


@pytest.mark.parametrize("N,queens", [
    (5, [(1, 3)]), (6, [(0, 1), (1, 3)]), (9, [(3, 0), (4, 2), (5, 4), (6, 6)]),
    (12, [(4, 1), (5, 3), (6, 5), (7, 7), (8, 9)]), (13, [(0, 0), (12, 11)]),
    (16, [(7, 0), (8, 2), (9, 4), (10, 6), (11, 8), (12, 10), (13, 12), (14, 14)]),
    (20, [(0, 19), (1, 17), (2, 15), (3, 13), (4, 11), (5, 9), (6, 7), (7, 5)])])
def test_neighbouring_rows(eng, oracle_mod, N, queens):
    want = oracle_mod.completions(N, [r for r, _ in queens], [c for _, c in queens])
    assert eng.count_completions(N, queens) == want


@pytest.mark.parametrize("N,queens", [
    (17, [(3, 4), (9, 11)]), (18, [(2, 2), (10, 7), (13, 16)]), (19, [(0, 3), (8, 12), (15, 5)]),   # attacked: none
    (19, [(0, 3), (8, 12), (15, 6)]),
    (27, [(26, 5), (18, 22), (12, 2), (13, 12), (19, 24), (14, 20), (23, 9), (16, 8)])])
def test_levels_over_the_gpu(eng, N, queens):
    """Two and three levels over the whole GPU, and a board whose top rows are free, where three do not fit the queue
    and two are counted: the counts of the same queries built as a batch."""
    from nqueens import CompletionJob
    b = eng.batch([CompletionJob(N, queens)])
    try:
        want = b.run()[0]
    finally:
        b.close()
    assert eng.count_completions(N, queens) == int(want)


def test_queries_beside_an_asynchronous_count(eng, oracle_mod):
    """A query has its own stream and buffers: one issued while an asynchronous count is outstanding leaves that
    count's result and status alone."""
    torch = pytest.importorskip("torch")
    import numpy as np
    import nqueens
    recs = nqueens.gen_records(17)
    d_rec = torch.from_numpy(recs.view(np.uint8).copy()).cuda()
    d_tot = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    eng.exec_device(17, d_rec.data_ptr(), len(recs), int((recs["startijkl"] >> 20).min()), d_tot.data_ptr())
    assert eng.count_completions(12, []) == 14200
    eng.sync()
    assert int(d_tot.item()) == oracle_mod.EXPECTED_TOTAL[17]
