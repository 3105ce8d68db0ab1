"""Boards that keep RA in rd, in one batch with boards whose words carry it.

A word's RA field lies at the board's last columns, so in a small board's word it would stand on the flags of the low
bits: only boards too large to keep RA in rd have it in their words.
"""
import numpy as np
import pytest

from conftest import gpu_available

COUNT = 1 << 5                  # the count flag of the device's compact words


def ra_in_rd(N, preset):
    return 2 * N - 5 - (preset - 3) <= 31


@pytest.mark.parametrize("N,preset", [(n, p) for n in range(19, 28) for p in (4, 5, 6)])
def test_words_that_carry_ra_leave_the_count_flag_alone(N, preset):
    import nqueens
    from test_native_cpu import schedule_of
    n = nqueens.lib().nq_start_constellations(N, None, 0)
    recs = np.concatenate([nqueens.gen_records_starts(N, f, 1, preset)[::37] for f in range(0, n, max(1, n // 40))])
    words = [w for r in recs[::max(1, len(recs) // 400)] for w in schedule_of(r, N)[2]]
    assert words and (ra_in_rd(N, preset) or not any(w & COUNT for w in words))


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("large", [(19, 4), (20, None)])
def test_small_boards_beside_a_large_one(oracle_mod, large):
    """Every count alone and beside a board whose words carry RA, at presets down to 4, with queries of both forms."""
    import nqueens
    C, Q = nqueens.CountJob, nqueens.CompletionJob
    small = [C(6, 4), C(6, 5), C(7, 4), C(8, 4), C(9, 4), C(10, 5), C(12, 4), C(13), C(16, 6), C(18)]
    for queries in ([], [Q(2, []), Q(3, [(0, 0)]), Q(5, []), Q(9, [(3, 0)]), Q(14, [(3, 3)])],
                    [Q(13, [(4, 1), (5, 3), (6, 5), (7, 7), (8, 9)])]):
        eng = nqueens.Engine(0, auto_tune=False)
        try:
            want = [oracle_mod.EXPECTED_TOTAL[j.N] for j in small]
            want += [oracle_mod.completions(q.N, [r for r, _ in q.queens], [c for _, c in q.queens]) for q in queries]
            b = eng.batch(small + queries + [C(*large)])
            try:
                got = b.run()
            finally:
                b.close()
            assert [int(x) for x in got] == want + [oracle_mod.EXPECTED_TOTAL[large[0]]]
        finally:
            eng.close()
