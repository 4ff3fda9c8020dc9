"""The model's rows are checked on the device: the first bad row decides the
error, wherever it stands, and nothing of a refused call remains.  Row counts
around the layer-1 tiles (64 rows), the GEMM's (128) and the inference chunk
(65536)."""
import numpy as np
import pytest

import lbm_oracle
import slide
import train_lb

pytestmark = pytest.mark.gpu

ARG, NOT_PERMUTATION = -1, -2


def _rows(width, n):
    rng = np.random.default_rng(n)
    return train_lb.vector_walks(width, n, 30, 60, n), rng.integers(0, 8, n).astype(np.int32)


@pytest.mark.parametrize("width", [4, 5])
@pytest.mark.parametrize("n", [1, 63, 65, 128, 129, 4000, 65536 + 130])
def test_predictions_of_every_row_count(width, n):
    tiles, slack = _rows(width, n)
    with slide.Solver(width, "manhattan") as s:
        s.lbm_init(5)
        got = s.lbm_predict(tiles, slack)
        pick = np.unique(np.concatenate([np.arange(min(n, 200)), np.arange(max(0, n - 200), n)]))
        want = lbm_oracle.predict(s.lbm_export(), tiles[pick], slack[pick], width)
        # relative to the predictions' spread, as in the gradient tests
        assert np.linalg.norm(got[pick] - want) <= 2e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("width", [4, 5])
@pytest.mark.parametrize("n,rows", [(128, (0, 5)), (384, (127, 128)), (384, (383, 383)), (65536 + 128, (65535, 65600)),
                                    (65536 + 128, (65536, 65537))])
@pytest.mark.parametrize("first", ["slack", "tiles"])
def test_first_bad_row_decides(width, n, rows, first):
    tiles, slack = _rows(width, n)
    a, b = rows
    if first == "slack":  # a row's slack is looked at before its tiles
        slack[a] = 256
        tiles[b] = 0
        want = ARG
    else:
        tiles[a, 0] = tiles[a, 1]
        slack[b if b > a else a] = -1
        want = NOT_PERMUTATION if b > a else ARG
    with slide.Solver(width, "manhattan") as s:
        s.lbm_init(5)
        before = s.lbm_export()
        out = np.full(n, 7.0, np.float32)
        st = s.lib.sp_lbm_predict(s.h, tiles.ctypes.data, slack.ctypes.data, n, out.ctypes.data)
        assert st == want and np.all(out == 7.0)
        if n <= 384:
            target = np.zeros(n, np.float32)
            for call in (lambda: s.lbm_train_step(tiles, slack, target, 1e-3),
                         lambda: s.lbm_gradients(tiles, slack, target)):
                with pytest.raises(slide.SlideError) as e:
                    call()
                assert e.value.status == want
            assert np.array_equal(s.lbm_export(), before)
            good, gs = _rows(width, n)
            s.lbm_train_step(good, gs, target, 1e-3)
            with slide.Solver(width, "manhattan") as t:  # the refused step did not count
                t.lbm_init(5)
                t.lbm_train_step(good, gs, target, 1e-3)
                d = np.abs(s.lbm_export() - t.lbm_export())
                assert np.quantile(d, 0.99) <= 1e-6  # summation order alone
