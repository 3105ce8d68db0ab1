"""The DFS lane's step as the kernel runs it: the child always becomes the current frame, the frame is saved with its
remaining candidates, and a sentinel frame under the stack feeds a lane without work.

The CPU test replays it in rounds of the kernel's length against the oracle and asserts what keeps its shared-memory
accesses in bounds; the GPU test counts short record lists per record at every split depth.
"""
import numpy as np
import pytest

from conftest import gpu_available

M32 = 0xFFFFFFFF
STEPS = 30                      # steps between two checks for finished lanes
SENTINEL_AVAIL, SENTINEL_WORD = 0xFFFFFFFE, M32


@pytest.fixture(scope="module")
def nq():
    import nqueens
    nqueens.lib()
    return nqueens


def _popc(x):
    return bin(x).count("1")


def replay(root, info, words):
    """Weighted count of one task: rounds of STEPS steps until the lane is idle at a check."""
    T, wexp, cnt, N = info & 31, (info >> 5) & 3, (info >> 7) & 1, (info >> 8) & 31
    if T == 31:
        return cnt << wexp
    ld, rd, col, avail = root
    fr = ((1 << N) - 1) & ~col
    R = _popc(fr)
    if T + 2 > R:
        return cnt << wexp
    tf, ram = R - T, 3 << (N - 1)
    words = [w ^ (1 << 28) for w in words[:T + 1]] + [SENTINEL_WORD]
    slots = [None] * (T + 2)
    slots[0] = (1, 0, (1 << (tf - 1)) - 1, SENTINEL_AVAIL)
    sp = 1
    for _ in range(100000):
        if avail == 0 and sp == 1:
            return cnt << wexp
        for _ in range(STEPS):
            if avail == 0:
                sp -= 1
                assert sp >= 0                       # the sentinel never runs out within a round
                ld, rd, fr, avail = slots[sp]
            d = R - _popc(fr)
            assert 0 <= d <= T + 1                   # the word read is the schedule's or the sentinel's
            bit = avail & -avail & M32
            rest = avail - bit
            w = words[d]
            s = w & 31
            assert sp < len(slots)
            slots[sp] = (ld, rd, fr, rest)
            sp += rest != 0
            x, y = (ld + bit) & M32, ((rd + bit) & M32) | (w & ram)
            nld = ((x << 32 | w) << s >> 32) & M32
            nrd = y >> s
            free = (fr - bit) & M32
            nf = free & ~(nld | nrd) & M32
            ahead = free & ~(((nld + nld) & M32) | (nrd >> 1)) & M32
            term = R - d == tf
            assert not (d == T + 1 and nf)           # the sentinel's children die
            cnt += term and nf != 0
            ld, rd, fr = nld, nrd, free
            avail = nf if nf and (ahead | (w & (1 << 28))) and not term else 0
    raise AssertionError("the lane does not end")


def _oracle_records(nq, oracle_mod, N, preset):
    o = oracle_mod.gen_constellations(N, preset)
    rec = np.zeros(len(o), nq.RECORD_DTYPE)
    rec["ld"] = o.ld & M32; rec["rd"] = o.rd & M32; rec["col"] = o.col & M32; rec["startijkl"] = o.startijkl
    return o, rec


@pytest.mark.parametrize("N,preset", [(7, 4), (9, 5), (11, 4), (12, 6), (13, 5)])
def test_lane_rounds_match_oracle(nq, oracle_mod, N, preset):
    from test_native_cpu import schedule_of
    o, rec = _oracle_records(nq, oracle_mod, N, preset)
    sol = oracle_mod.exec_solutions(N, o, threads=1)
    for i in range(0, len(rec), max(1, len(rec) // 400)):
        assert replay(*schedule_of(rec[i], N)) == int(sol[i]), (i, rec[i])


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("split", [0, 1, 2, 3])
@pytest.mark.parametrize("N,m", [(8, 1), (12, 33), (14, 5), (15, 700), (16, 3)])
def test_short_lists_per_record(nq, oracle_mod, N, m, split):
    """Lists much shorter than the grid's lanes, per record against the oracle, at every split depth and block."""
    o, rec = _oracle_records(nq, oracle_mod, N, 5)
    at = np.sort(np.random.default_rng(100 * N + m).choice(len(rec), m, replace=False))
    want = oracle_mod.exec_solutions(N, oracle_mod.Records(o.ld[at], o.rd[at], o.col[at], o.startijkl[at]))
    eng = nq.Engine(0, auto_tune=False)
    try:
        for block in (64, 128, 256):
            eng.set_config(block, 0, split)
            total, sol = eng.exec_records(N, np.ascontiguousarray(rec[at]), want_solutions=True)
            assert np.array_equal(sol, want), (block, split)
            assert total == int(want.sum())
    finally:
        eng.close()


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("grid", [1, 3, 0])
@pytest.mark.parametrize("m", [1, 31, 1000])
def test_shared_work_counts_every_solution_once(nq, oracle_mod, m, grid):
    """Few large items: lanes of a warp give parts of them to each other (grid 1 and 3: the pool is refilled in
    chunks too).  Every record's count, in which several lanes take part, equals the oracle's."""
    N = 15
    o, rec = _oracle_records(nq, oracle_mod, N, 4)
    at = np.sort(np.random.default_rng(m).choice(len(rec), m, replace=False))
    want = oracle_mod.exec_solutions(N, oracle_mod.Records(o.ld[at], o.rd[at], o.col[at], o.startijkl[at]))
    eng = nq.Engine(0, auto_tune=False)
    try:
        for split in (0, 2):
            eng.set_config(64, grid, split)
            total, sol = eng.exec_records(N, np.ascontiguousarray(rec[at]), want_solutions=True)
            assert np.array_equal(sol, want), (m, grid, split)
            assert total == int(want.sum())
    finally:
        eng.close()
