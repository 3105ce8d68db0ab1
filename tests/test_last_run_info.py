"""The queue's length right after an asynchronous call, short lists and long, on both streams."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("N,m,split", [(9, 392, -1), (14, 12289, -1), (14, 5000, 0), (14, 5000, 3), (17, 20000, -1)])
def test_queue_length_before_the_wait(N, m, split):
    import nqueens
    torch = pytest.importorskip("torch")
    r = np.ascontiguousarray(nqueens.gen_records(N)[:m])
    start = int((r["startijkl"] >> 20).min())
    d_rec = torch.from_numpy(r.view(np.int32).copy()).cuda()
    d_total = torch.zeros(1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        eng.set_config(64, 0, split)
        total = eng.exec_records(N, r)[0]
        want = eng.last_run_info()
        assert want[1] == len(r) if want[0] == 0 else want[1] > len(r)
        for stream in (0, side.cuda_stream):
            eng.exec_records(N, r[:50])                       # another length in between
            eng.exec_device(N, d_rec.data_ptr(), len(r), start, d_total.data_ptr(), 0, stream)
            assert eng.last_run_info() == want
            eng.sync()
            assert eng.last_run_info() == want and int(d_total.item()) == total
    finally:
        eng.close()
