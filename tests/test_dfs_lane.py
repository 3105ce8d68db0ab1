"""The DFS lane's step as the kernel runs it: the child always becomes the current frame, the frame is saved with its
remaining candidates, a solution is a frame in the base row, and a sentinel frame under the stack feeds a lane without
work.

The CPU test replays it in rounds of the kernel's length against the oracle, with RA in rd and in the words, and asserts
what keeps its shared-memory accesses in bounds; the GPU tests count short record lists per record at every split depth.
"""
import numpy as np
import pytest

from conftest import gpu_available

M32 = 0xFFFFFFFF
STEPS = 30                      # steps between two checks for finished lanes
SENTINEL_AVAIL, COUNT_WORD = 0xFFFFFFFE, M32
NOLOOK, COUNT = 1 << 28, 1 << 5


@pytest.fixture(scope="module")
def nq():
    import nqueens
    nqueens.lib()
    return nqueens


def _popc(x):
    return bin(x).count("1")


def replay(root, info, words, ra_words):
    """Weighted count of one task: rounds of STEPS steps until the lane is idle at a check."""
    T, wexp, cnt, N = info & 31, (info >> 5) & 3, (info >> 7) & 1, (info >> 8) & 31
    if T == 31:
        return cnt << wexp
    ld, rd, col, avail = root
    fr = ((1 << N) - 1) & ~col
    R = _popc(fr)
    assert R == T + 2                                # one column left in the base row
    tf, ram = R - T, 3 << (N - 1)
    words = [w ^ NOLOOK for w in words[:T + 1]]
    if not ra_words:                                 # RA above the board in rd, as many places up as rows follow
        rows = 0
        for d, w in enumerate(words):
            rows += w & 31
            rd |= ((w & ram) >> (w & 31)) << rows
            words[d] = w & ~ram
        assert rd <= M32
        ram = 0
    assert not any(w & COUNT for w in words) or N < 7
    words.append(COUNT_WORD)
    slots = [None] * (T + 3)
    slots[0] = (1, 0, (1 << (tf - 1)) - 1, SENTINEL_AVAIL)
    sp = 1
    for _ in range(100000):
        if avail == 0 and sp == 1:
            return (cnt - (31 - _popc(slots[0][3]))) << wexp
        for _ in range(STEPS):
            if avail == 0:
                sp -= 1
                assert sp >= 0                       # the sentinel never runs out within a round
                ld, rd, fr, avail = slots[sp]
            d = R - _popc(fr)
            assert 0 <= d <= T + 1                   # the word read is the schedule's or the count word
            rest = avail & (avail - 1)
            bit = avail - rest
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
            assert d <= T or not nf                  # the count word's children die
            cnt += bool(w & COUNT)
            ld, rd, fr = nld, nrd, free
            avail = nf if ahead | (w & NOLOOK) else 0
    raise AssertionError("the lane does not end")


def _oracle_records(nq, oracle_mod, N, preset):
    o = oracle_mod.gen_constellations(N, preset)
    rec = np.zeros(len(o), nq.RECORD_DTYPE)
    rec["ld"] = o.ld & M32; rec["rd"] = o.rd & M32; rec["col"] = o.col & M32; rec["startijkl"] = o.startijkl
    return o, rec


@pytest.mark.parametrize("N,preset", [(6, 4), (7, 4), (9, 5), (11, 4), (12, 6), (13, 5)])
def test_lane_rounds_match_oracle(nq, oracle_mod, N, preset):
    from test_native_cpu import schedule_of
    o, rec = _oracle_records(nq, oracle_mod, N, preset)
    sol = oracle_mod.exec_solutions(N, o, threads=1)
    for i in range(0, len(rec), max(1, len(rec) // 400)):
        for ra_words in (False, True) if N > 7 else (False,):
            assert replay(*schedule_of(rec[i], N), ra_words) == int(sol[i]), (i, rec[i])


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


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("split", [0, 1])
def test_records_with_columns_to_spare(nq, oracle_mod, split):
    """Records no generator makes, with used columns cleared: more columns than rows are left, and a base row counts
    once whatever it has free (dfs_iter's rule).  Per record against the oracle, among regular records."""
    N = 11
    o, rec = _oracle_records(nq, oracle_mod, N, 5)
    at = np.arange(0, len(rec), 37)
    col = o.col[at].copy()
    rng = np.random.default_rng(3)
    for i in range(0, len(at), 2):
        used = [b for b in range(2, N - 1) if int(col[i]) >> b & 1]
        if used:
            col[i] = np.uint64(int(col[i]) & ~(1 << used[rng.integers(len(used))]))
    want = oracle_mod.exec_solutions(N, oracle_mod.Records(o.ld[at], o.rd[at], col, o.startijkl[at]))
    r = np.ascontiguousarray(rec[at])
    r["col"] = col & M32
    eng = nq.Engine(0, auto_tune=False)
    try:
        eng.set_config(64, 0, split)
        total, sol = eng.exec_records(N, r, want_solutions=True)
        assert np.array_equal(sol, want)
    finally:
        eng.close()
