"""Whole-board counts from lists generated on the device: every preset it takes against the known totals and the host
generator's record numbers, and ranges whose records take several buffers."""
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")]


@pytest.fixture(scope="module")
def eng():
    import nqueens
    e = nqueens.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("N,preset", [(6, 4), (7, 5), (8, 6), (9, 4), (10, 8), (12, 7), (13, 6), (15, 4), (15, 8),
                                      (16, 5), (17, 6), (18, 4)])
def test_presets(eng, oracle_mod, N, preset):
    import nqueens
    try:
        want = len(nqueens.gen_records(N, preset))
    except nqueens.NQError as e:
        with pytest.raises(nqueens.NQError) as got:
            eng.count(N, preset)
        assert got.value.status == e.status
        return
    total = eng.count(N, preset).total
    assert eng.last_count_info()[1] == want
    if want and preset <= 5:
        assert total == oracle_mod.EXPECTED_TOTAL[N]
    if want:
        eng.set_chunk_records(max(1, want // 3))          # the host-generated list
        try:
            assert eng.count(N, preset).total == total
        finally:
            eng.set_chunk_records(0)


def test_start_ranges_of_a_large_board(eng):
    """N=22, preset 7: ranges generated on the device add up to the host-generated count of their union."""
    import nqueens
    a = [eng.count_starts(22, f, 4) for f in (9000, 9004)]
    recs = nqueens.gen_records_starts(22, 9000, 8)
    assert sum(a) == eng.exec_records(22, recs)[0]
