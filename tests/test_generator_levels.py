"""Counts of single start constellations on small boards, where a level between may hold more states than there are
records: the device's list against the host's, preset by preset."""
import pytest

from conftest import gpu_available


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("N,preset", [(6, 7), (6, 8), (7, 6), (7, 7), (7, 8), (8, 8), (9, 8)])
def test_single_starts(N, preset):
    import nqueens
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        for f in range(len(nqueens.start_constellations(N))):
            try:
                recs = nqueens.gen_records_starts(N, f, 1, preset)
                want = eng.exec_records(N, recs)[0] if len(recs) else 0
            except nqueens.NQError as e:
                with pytest.raises(nqueens.NQError) as got:
                    eng.count_starts(N, f, 1, preset)
                assert got.value.status == e.status
                continue
            assert eng.count_starts(N, f, 1, preset) == want
            assert eng.last_count_info()[1] == len(recs)
    finally:
        eng.close()
