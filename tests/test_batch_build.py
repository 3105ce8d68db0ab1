"""Batches built on the device: jobs that share a board, queries of both word forms, settled jobs and a host-made list in
one batch give each job's count alone, in one launch, from a graph and job by job."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


def _jobs(kind):
    from nqueens import CompletionJob as Q, CountJob as C
    if kind == "boards":
        return [C(12), C(6), C(12), C(13, 6), C(12, 4), C(13, 9), C(16), C(16)]
    if kind == "small":
        return [C(1), C(2), C(3), C(4), C(5), Q(4, [(0, 1)]), Q(8, [(0, 0), (1, 1)]), Q(3, [(0, 0), (2, 1)]),
                Q(4, [(2, 0), (0, 1), (3, 2), (1, 3)])]
    if kind == "compact":
        return [Q(14, [(3, 3)]), Q(13, []), C(13), Q(15, [(0, 7), (14, 6)]), Q(14, [(3, 3)])]
    return [Q(14, [(4, 1), (5, 3), (6, 5), (7, 7), (8, 9)]), C(13), Q(18, [(2, 17), (9, 8), (10, 5)]), Q(5, []), C(13)]


@pytest.mark.parametrize("split", [-1, 0, 2])
@pytest.mark.parametrize("kind", ["boards", "small", "compact", "wide"])
def test_batch_equals_each_job_alone(kind, split):
    import nqueens
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        eng.set_config(64, 0, split)
        jobs = _jobs(kind)
        want = np.array([eng.count(j.N, j.preset).total if isinstance(j, nqueens.CountJob) else
                         eng.count_completions(j.N, j.queens) for j in jobs], np.uint64)
        b = eng.batch(jobs)
        try:
            assert np.array_equal(b.run(use_graph=False), want)
            assert np.array_equal(b.run(use_graph=True), want)
            assert np.array_equal(b.run_plain(), want)
            assert b.device_bytes <= sum(eng.job_device_bytes(j) for j in jobs)
        finally:
            b.close()
    finally:
        eng.close()


def test_batch_rejects_a_preset_too_deep():
    import nqueens
    eng = nqueens.Engine(0)
    try:
        for job, status in ((nqueens.CountJob(10, 3), -6), (nqueens.CompletionJob(8, [(3, 3), (3, 3)]), -1)):
            with pytest.raises(nqueens.NQError) as e:
                eng.batch([nqueens.CountJob(9), job])
            assert e.value.status == status
    finally:
        eng.close()


@pytest.mark.parametrize("n", [1, 15, 254, 255, 2048, 2049])
def test_totals_of_many_jobs(oracle_mod, n):
    """Numbers of jobs on both sides of the read-back's rules: every total, run after run."""
    import nqueens
    eng = nqueens.Engine(0, auto_tune=False)
    sizes = [6 + (i * 7 + i // 5) % 4 for i in range(n)]
    try:
        b = eng.batch([nqueens.CountJob(N) for N in sizes])
        try:
            for use_graph in (False, True, True):
                assert list(b.run(use_graph=use_graph)) == [oracle_mod.EXPECTED_TOTAL[N] for N in sizes]
        finally:
            b.close()
    finally:
        eng.close()


def test_batches_from_two_threads_give_their_memory_back(oracle_mod):
    """Batches of all sizes built, run and released by two threads at once on one handle, one of them larger than what
    the handle keeps between batches: right counts, and the device's memory is free again after the handle."""
    import threading
    import nqueens
    torch = pytest.importorskip("torch")
    wrong = []

    def work(eng, sizes):
        for N, n in sizes:
            b = eng.batch([nqueens.CountJob(N)] * n)
            try:
                if list(b.run(use_graph=False)) != [oracle_mod.EXPECTED_TOTAL[N]] * n:
                    wrong.append((N, n))
            finally:
                b.close()

    def cycle():
        eng = nqueens.Engine(0, auto_tune=False)
        try:
            threads = [threading.Thread(target=work, args=(eng, s))
                       for s in ([(8, 3), (13, 40), (15, 24), (9, 100)], [(12, 64), (10, 2), (14, 20), (11, 9)])]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
        finally:
            eng.close()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    first = cycle()
    assert cycle() >= first - (8 << 20) and not wrong


@pytest.mark.parametrize("sizes", [[13, 14, 15], [15] * 9 + [13], [16, 15] * 12, [14] * 40 + [16], [17, 16, 14, 13]])
def test_unsplit_boards_in_a_batch(oracle_mod, sizes):
    """Batches on both sides of the rule for unsplit boards, mixed with boards that are split."""
    import nqueens
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        b = eng.batch([nqueens.CountJob(N) for N in sizes])
        try:
            want = [oracle_mod.EXPECTED_TOTAL[N] for N in sizes]
            assert list(b.run(use_graph=False)) == want and list(b.run_plain()) == want
            assert b.device_bytes <= sum(eng.job_device_bytes(nqueens.CountJob(N)) for N in sizes)
        finally:
            b.close()
    finally:
        eng.close()


@pytest.mark.parametrize("n", [64, 65])
def test_many_queries_with_counts(n):
    """On both sides of the number of queries from which each starts from fewer frames and is split further."""
    import random
    import nqueens
    rng = random.Random(7)
    jobs = [nqueens.CountJob(N) for N in (16, 15, 16)]
    for _ in range(n):
        N, k = rng.randint(9, 16), rng.randint(1, 3)
        jobs.append(nqueens.CompletionJob(N, list(zip(rng.sample(range(N), k), rng.sample(range(N), k)))))
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        want = [eng.count(j.N).total if isinstance(j, nqueens.CountJob) else eng.count_completions(j.N, j.queens) for j in jobs]
        b = eng.batch(jobs)
        try:
            assert list(b.run(use_graph=False)) == want and list(b.run(use_graph=True)) == want
        finally:
            b.close()
    finally:
        eng.close()
