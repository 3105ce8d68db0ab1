"""Short calls whose launches follow each other without a read-back: the counts come from the last block of the search,
the times from the device's clock, and each call leaves the handle ready for any other."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("N,m", [(6, 5), (8, 1), (10, 1007), (13, 7731), (16, 16384), (16, 33046), (17, 16384), (17, 16385)])
def test_same_counts_with_and_without_read_back(N, m):
    import nqueens
    r = np.ascontiguousarray(nqueens.gen_records(N)[:m])
    eng = nqueens.Engine(0)
    try:
        got = eng.exec_records(N, r, want_solutions=True)
        prep, dfs = eng.last_kernel_ms()
        assert 0 <= prep < 1e3 and 0 < dfs < 1e3
        eng.set_queue_order(1)                     # reads the queue's length between its launches
        want = eng.exec_records(N, r, want_solutions=True)
        assert got[0] == want[0] == int(np.sum(got[1])) and np.array_equal(got[1], want[1])
    finally:
        eng.close()


def test_calls_of_every_kind_in_turn(oracle_mod):
    import nqueens
    import torch
    total, unique = oracle_mod.EXPECTED_TOTAL, oracle_mod.EXPECTED_UNIQUE
    r = nqueens.gen_records(12)
    start = int((r["startijkl"] >> 20).min())
    d_rec = torch.from_numpy(r.view(np.int32).copy()).cuda()
    d_total = torch.zeros(1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    eng = nqueens.Engine(0)
    try:
        for N in (9, 17, 11, 6, 14):               # 17: the list is long enough for a read-back
            for stream in (0, side.cuda_stream):
                eng.exec_device(12, d_rec.data_ptr(), len(r), start, d_total.data_ptr(), 0, stream)
                assert eng.count_completions(N, []) == total[N]      # a stream of its own, while the list runs
                eng.sync()
                assert eng.last_kernel_ms()[1] > 0 and int(d_total.item()) == total[12]
            assert eng.count(N).total == total[N]
            u = eng.count_unique(N)
            assert (u.unique, u.total) == (unique[N], total[N])
            assert eng.exec_records(12, r)[0] == total[12]
    finally:
        eng.close()


def test_a_capturing_stream_is_refused(oracle_mod):
    """A call on a stream under capture fails with a status, short lists included, and the handle goes on."""
    import nqueens
    import torch
    r = nqueens.gen_records(10)
    start = int((r["startijkl"] >> 20).min())
    d_rec = torch.from_numpy(r.view(np.int32).copy()).cuda()
    d_total = torch.zeros(1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            with pytest.raises(nqueens.NQError) as e:
                eng.exec_device(10, d_rec.data_ptr(), len(r), start, d_total.data_ptr(), 0, side.cuda_stream)
            d_total.add_(1)
        assert e.value.status == -4
        eng.exec_device(10, d_rec.data_ptr(), len(r), start, d_total.data_ptr(), 0, side.cuda_stream)
        eng.sync()
        assert int(d_total.item()) == oracle_mod.EXPECTED_TOTAL[10]
    finally:
        eng.close()
