"""What a board's list takes: its exact numbers of states size the device generator's buffers and the batches, and a
request is admitted by what it needs, not by a bound of several times that."""
import numpy as np
import pytest

from conftest import gpu_available

MIB = 1 << 20


def _widest(N, preset):
    """The widest level from the start constellations to the records.  A corner start (j = N - 1) holds three queens,
    the others four, and a level adds one to those below the preset."""
    import nqueens

    def split(q):
        r = nqueens.gen_records(N, q)
        corner = int(np.count_nonzero((r["startijkl"] >> 10 & 31) == N - 1))
        return len(r) - corner, corner
    starts = nqueens.start_constellations(N)
    corners = {3: int(np.count_nonzero((np.asarray(starts) >> 10 & 31) == N - 1))}
    sides = {}
    for q in range(4, preset + 1):
        sides[q], corners[q] = split(q)
    return max(sides[min(preset, 4 + lv)] + corners[3 + lv] for lv in range(preset - 2))


@pytest.mark.parametrize("N,preset", [(n, p) for n in range(6, 16) for p in (4, 5, 6, 7, 8) if (n, p) != (7, 8)] +
                         [(16, 6), (17, 5), (18, 6), (19, 6), (20, 6), (22, 5), (24, 5), (27, 4), (27, 5)])
def test_states_of_every_board(N, preset):
    import nqueens
    got = nqueens.lib().nq_debug_board_states(N, preset)
    assert got == _widest(N, preset)
    if N >= 12:
        assert got == len(nqueens.gen_records(N, preset))


def test_states_outside_the_device_generator():
    import nqueens
    f = nqueens.lib().nq_debug_board_states
    assert [f(5, 5), f(28, 5), f(12, 3), f(12, 9)] == [0] * 4
    with pytest.raises(nqueens.NQError) as e:
        nqueens.engine.job_device_bytes(nqueens.CountJob(7, 8), 152)      # too deep: refused before it is built
    assert e.value.status == -6


@pytest.mark.parametrize("N,limit", [(12, 440 << 10), (14, 160 * MIB), (16, 52 * MIB), (17, 77 * MIB), (18, 160 * MIB),
                                     (19, 254 * MIB), (20, 392 * MIB), (21, 588 * MIB), (22, 8327 * MIB), (23, 13005 * MIB)])
def test_counts_are_admitted_by_their_records(N, limit):
    """A task's record, root, info, schedule of 4-byte words and queue items: a budget of 16 GiB takes N=23, of 1 GiB
    N=21."""
    import nqueens
    assert nqueens.engine.job_device_bytes(nqueens.CountJob(N), 152) <= limit


@pytest.mark.parametrize("N,k", [(8, 0), (12, 2), (16, 0), (18, 2), (20, 3), (22, 1), (27, 4)])
def test_queries_are_sized_by_their_rows(N, k):
    import nqueens
    q = [(3 * i, (7 * i + 2) % N) for i in range(k)]
    size = nqueens.engine.job_device_bytes(nqueens.CompletionJob(N, q), 152)
    assert size < 64 * MIB
    if N <= 12:
        assert size < 2 * MIB


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("jobs", [[(13, 8), (14, 7)], [(16, 7)], [(11, 8), (10, 7), (9, 7), (8, 6), (6, 7)],
                                  [(17, 5), (12, 6), (18, 4)]])
def test_deep_presets_alone_and_in_a_batch(oracle_mod, jobs):
    """Lists the device makes for deep presets: the number of records and the count, alone and beside others."""
    import nqueens
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        want = []
        for N, p in jobs:
            n = len(nqueens.gen_records(N, p))
            want.append(eng.count(N, p).total)
            assert eng.last_count_info()[1] == n
            eng.set_chunk_records(max(1, n // 2 + 1))           # the host's list
            assert eng.count(N, p).total == want[-1]
            eng.set_chunk_records(0)
            if p <= 5:
                assert want[-1] == oracle_mod.EXPECTED_TOTAL[N]
        queries = [nqueens.CompletionJob(14, [(3, 3)]), nqueens.CompletionJob(10, [(0, 2), (5, 5)])]
        want += [eng.count_completions(q.N, q.queens) for q in queries]
        for order in (1, -1):
            cs = ([nqueens.CountJob(N, p) for N, p in jobs] + queries)[::order]
            b = eng.batch(cs)
            try:
                assert [int(x) for x in b.run()][::order] == want
                assert b.device_bytes <= sum(eng.job_device_bytes(j) for j in cs)
            finally:
                b.close()
    finally:
        eng.close()
