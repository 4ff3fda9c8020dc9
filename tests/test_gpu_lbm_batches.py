"""Gradients at the batch sizes where the GEMMs' split changes: one K chunk
pair, fewer chunks than split CTAs, a ragged last share."""
import numpy as np
import pytest

import lbm_oracle
import slide
import train_lb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [4, 5])
@pytest.mark.parametrize("n", [128, 384, 3328, 6528, 8320])
def test_gradients(width, n):
    rng = np.random.default_rng(n)
    tiles = train_lb.vector_walks(width, n, 30, 60, n)
    slack = rng.integers(0, 8, n).astype(np.int32)
    target = (3.0 * slack + rng.normal(0, 2, n)).astype(np.float32)
    with slide.Solver(width, "manhattan") as s:
        s.lbm_init(7)
        params = s.lbm_export()
        loss, grads = s.lbm_gradients(tiles, slack, target)
        want_loss, _, want = lbm_oracle.forward_backward(params, tiles, slack, target, width)
        assert abs(loss - want_loss) <= 2e-3 * want_loss
        # per parameter group, as in the model's gradient test
        for name, a, b in zip(("W1", "b1", "W2", "b2", "w3", "b3"), lbm_oracle.split(grads.astype(np.float64), width),
                              lbm_oracle.split(want, width)):
            assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b), name
        # a step along them changes every group the gradient is not zero in
        s.lbm_train_step(tiles, slack, target, 1e-3)
        moved = s.lbm_export() - params
        assert np.all((np.abs(moved) > 0) == (np.abs(grads) > 0)) or np.mean((moved != 0) == (grads != 0)) > 0.999
