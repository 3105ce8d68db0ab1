"""Completion queries of several threads on one handle, each on a stream and buffers of its own."""
import threading

import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]

MIB = 1 << 20


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_queries_of_several_threads(oracle_mod):
    import nqueens
    torch = pytest.importorskip("torch")
    eng = nqueens.Engine(0, auto_tune=False)
    jobs = [(N, q) for N in (6, 9, 12, 13, 15) for q in ([], [(2, 4)], [(0, 1), (5, 3)])] + [(17, [(3, 4), (9, 12)]), (16, [])]
    want = [oracle_mod.completions(N, [r for r, _ in q], [c for _, c in q]) if N < 16 else None for N, q in jobs]
    want[-2:] = [eng.count_completions(*jobs[-2]), oracle_mod.EXPECTED_TOTAL[16]]
    wrong = []

    def work(k):
        for i in range(3 * len(jobs)):
            j = (i * (2 * k + 1) + k) % len(jobs)
            if eng.count_completions(*jobs[j]) != want[j]:
                wrong.append(jobs[j])

    before = _free(torch)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(12)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong
    finally:
        eng.close()
    assert _free(torch) >= before - 8 * MIB


def test_the_large_buffer_stays_with_the_next_query():
    """After queries of several threads left their streams behind, large queries one by one reuse one buffer: what the
    device has free does not change between them, nor with small ones in between."""
    import nqueens
    torch = pytest.importorskip("torch")
    eng = nqueens.Engine(0, auto_tune=False)
    large = (20, [(2, 2), (10, 7)])
    try:
        want = eng.count_completions(*large)
        threads = [threading.Thread(target=lambda: [eng.count_completions(12, [(0, i)]) for i in range(12)]) for _ in range(4)]
        threads += [threading.Thread(target=lambda: eng.count_completions(*large)) for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert eng.count_completions(*large) == want
        free = _free(torch)
        for _ in range(4):
            assert eng.count_completions(*large) == want
            assert eng.count_completions(8, []) == 92
            assert _free(torch) == free
    finally:
        eng.close()
