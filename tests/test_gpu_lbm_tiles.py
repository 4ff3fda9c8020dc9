"""Predictions do not depend on how many tiles of rows a block of layer 1
streams: a call's rows in one piece, with padding after the last, and the same
rows in calls of one tile per block, bit for bit."""
import numpy as np
import pytest

import slide
import train_lb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [4, 5])
@pytest.mark.parametrize("n", [4865, 9729, 20033, 65536 + 4865])
def test_rows_in_one_call_and_in_many(width, n):
    rng = np.random.default_rng(n)
    tiles = train_lb.vector_walks(width, n, 30, 60, n)
    slack = rng.integers(0, 256, n).astype(np.int32)
    with slide.Solver(width, "manhattan") as s:
        s.lbm_init(9)
        whole = s.lbm_predict(tiles, slack)
        parts = [s.lbm_predict(tiles[a:a + 2048], slack[a:a + 2048]) for a in range(0, n, 2048)]
        assert np.array_equal(whole, np.concatenate(parts))
