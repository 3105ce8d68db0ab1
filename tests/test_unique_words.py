"""The unique counter's row rules as words: the columns of every row by backTrack1's and backTrack2's rules
(07Py_bit_symmetry.py:126-170), and the flags above them, for every start of every board."""
import numpy as np
import pytest

COUNT, CLASSIFY, NOLOOK, SIDES = 1 << 27, 1 << 28, 1 << 29, 1 << 31


def rules(N, part, bound1, lastmask, left):
    """Word of a frame with `left` rows left, its own included: its child stands in row N - left + 1."""
    if left == 0:
        return 0
    if left == 1:
        return COUNT if part == 1 else CLASSIFY
    child, bound2, side = N - left + 1, N - 1 - bound1, (1 << (N - 1)) | 1
    columns, flags = (1 << N) - 1, 0
    if left == 2:
        flags |= NOLOOK                       # no row behind the last one to look at
    if part == 1:
        if child < bound1:
            columns &= ~2
    else:
        if child < bound1:
            columns &= ~side
        if child == N - 1:
            columns &= ~lastmask
        if child == bound2 + 1:
            flags |= SIDES
    return columns | flags


@pytest.mark.parametrize("N", range(4, 28))
def test_row_words(N):
    from nqueens import _lib
    starts = [(1, b, 0) for b in range(2, N - 1)]
    lastmask = (1 << (N - 1)) | 1
    b = 1
    while b < N - 1 - b:
        starts.append((2, b, lastmask))
        lastmask |= (lastmask << 1) | (lastmask >> 1)
        b += 1
    words = np.zeros(32, np.uint32)
    for i, (part, bound1, mask) in enumerate(starts):
        assert _lib.lib().nq_debug_unique_words(N, i, _lib.p32(words)) == 0
        for left in range(N + 1):
            assert int(words[left]) == rules(N, part, bound1, mask, left), (part, bound1, left)
    assert _lib.lib().nq_debug_unique_words(N, len(starts), _lib.p32(words)) == -1
