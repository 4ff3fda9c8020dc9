"""sp_idas_parallel on rows that are no permutation, which it takes as they come:
two blanks, tiles twice, and no blank at all, where a move and its reverse do
not give the board back and the answer depends on the whole walk."""
import numpy as np
import pytest

import instances
from test_gpu_first_path import _gpu_rows, _reference_tables

pytestmark = pytest.mark.gpu

DELTA = (-4, 1, -1, 4)


def _walk(tiles, limit, hd, mv):
    """One root by one thread: the blank (the last cell with tile 0, cell 0
    without one) and the tile it meets are exchanged by xor, h by the table."""
    b = [int(t) & 15 for t in tiles]
    blank = max([c for c in range(16) if not b[c]], default=0)
    h = sum(abs(c // 4 - t // 4) + abs(c % 4 - t % 4) for c, t in enumerate(b) if t)
    path, d = [], 0

    def slide(d):
        nonlocal blank, h
        to = blank + DELTA[d]
        t = b[to]
        h += int(hd[t, to, d])
        b[to] ^= t
        b[blank] ^= t
        blank = to

    while True:
        if h == 0:
            return path
        if (not path or path[-1] != 3 - d) and mv[blank, d]:
            to = blank + DELTA[d]
            if len(path) + 1 + h + int(hd[b[to], to, d]) <= limit and len(path) < 251:
                slide(d)
                path.append(d)
                d = 0
                continue
        d += 1
        while d == 4:
            if not path:
                return None
            d = path.pop()
            slide(3 - d)
            d += 1


def _signs(mv):
    """A table of random signs whose reverse moves take back what the moves add."""
    rng = np.random.default_rng(7)
    hd = np.zeros((16, 16, 4), np.int8)
    for t in range(16):
        for c in range(16):
            for d in (0, 1):
                to = c - DELTA[d]
                if 0 <= to < 16 and mv[to, d]:
                    hd[t, c, d] = rng.choice([-1, 1])
                    hd[t, to, 3 - d] = -hd[t, c, d]
    return hd


@pytest.mark.parametrize("n", [1, 40, 305, 1100])
@pytest.mark.parametrize("limit", [6, 11])
@pytest.mark.parametrize("table", ["reference", "signs"])
def test_rows_that_are_no_permutation(n, limit, table):
    hd, mv = _reference_tables()
    if table == "signs":
        hd = _signs(mv)
    roots = np.concatenate([instances.random_walks(4, 1, 1 + i % 7, seed=i + n) for i in range(n)])
    rng = np.random.default_rng(n + limit)
    for i in range(0, n, 3):
        c = int(np.argmin(roots[i]))
        roots[i, c] = int(rng.integers(1, 16)) + 16 * int(rng.integers(0, 2))  # no blank
    for i in range(1, n, 3):
        roots[i, int(rng.integers(0, 16))] = 16 * int(rng.integers(0, 16))    # a blank more
    got = _gpu_rows(roots, limit, hd, mv)
    for i in range(n):
        want = _walk(roots[i], limit, hd, mv)
        assert int(got[i, 0]) == (-1 if want is None else len(want)), i
        if want:
            assert list(got[i, 1:1 + len(want)]) == want, i
