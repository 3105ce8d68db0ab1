"""Device memory of the unique counter: buffers for the states there are, and rows fewer where the device has no room."""
import pytest

from conftest import gpu_available

MIB = 1 << 20


def _levels(N, levels):
    """States after each expanded row, breadth first by the row rules of backTrack1 and backTrack2
    (07Py_bit_symmetry.py:126-170); a state in the last row but one, or below row 7, stays."""
    mask, side = (1 << N) - 1, (1 << (N - 1)) | 1
    cur = []

    def allowed(row, left, down, right, part, bound1):
        free = mask & ~(left | down | right)
        if part == 1:
            return free & ~2 if row < bound1 else free
        if row < bound1:
            return free & ~side
        if row == N - 1 - bound1:
            used = down & side
            return 0 if used == 0 else free if used == side else free & side
        return free

    starts = [(1, b) for b in range(2, N - 1)] + [(2, b) for b in range(1, N) if b < N - 1 - b]
    for part, b in starts:
        bit = 1 << b
        s = (2, (2 | bit) << 1, 1 | bit, (2 | bit) >> 1) if part == 1 else (1, bit << 1, bit, bit >> 1)
        if allowed(*s, part, b):
            cur.append((*s, part, b))
    out = [len(cur)]
    for _ in range(levels):
        nxt = []
        for s in cur:
            row, left, down, right, part, b = s
            if row + 1 >= N - 1 or row + 1 >= 8:
                nxt.append(s)
                continue
            free = allowed(*s)
            while free:
                bit = free & -free
                free ^= bit
                t = (row + 1, (left | bit) << 1, down | bit, (right | bit) >> 1, part, b)
                if allowed(*t):
                    nxt.append(t)
        cur = nxt
        out.append(len(cur))
    return out


@pytest.mark.parametrize("N,levels", [(n, 6) for n in range(4, 13)] + [(14, 5), (17, 4), (20, 3), (23, 3), (27, 3)])
def test_states_of_each_level(N, levels):
    import nqueens
    f = nqueens.lib().nq_debug_unique_states
    assert [f(N, l) for l in range(levels + 1)] == _levels(N, levels)
    assert f(3, 0) == f(28, 0) == f(N, 7) == -1


def _free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("N,most", [(4, 4), (9, 4), (12, 6), (15, 28), (16, 52), (17, 30), (18, 176)])
def test_a_board_takes_what_its_size_needs(oracle_mod, N, most):
    import nqueens
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    warm = nqueens.Engine(0, auto_tune=False)                   # loads the kernels
    warm.count_unique(N)
    warm.close()
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        before = _free(torch)
        r = eng.count_unique(N)
        assert (r.unique, r.total) == (oracle_mod.EXPECTED_UNIQUE[N], oracle_mod.EXPECTED_TOTAL[N])
        assert before - _free(torch) <= most * MIB
    finally:
        eng.close()


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="needs a CUDA GPU")
def test_a_device_with_little_room_left(oracle_mod):
    """Beside a reservation of nearly all of the device's memory N=18 runs from the row before, N=16 as ever."""
    import nqueens
    torch = pytest.importorskip("torch")
    eng = nqueens.Engine(0, auto_tune=False)
    eng.count_unique(18)
    eng.close()
    eng = nqueens.Engine(0, auto_tune=False)
    try:
        hog = torch.empty(_free(torch) - 96 * MIB, dtype=torch.uint8, device="cuda")
        assert _free(torch) < 128 * MIB
        for N in (16, 18, 17):
            r = eng.count_unique(N)
            assert (r.unique, r.total) == (oracle_mod.EXPECTED_UNIQUE[N], oracle_mod.EXPECTED_TOTAL[N])
        del hog
    finally:
        eng.close()
        torch.cuda.empty_cache()
