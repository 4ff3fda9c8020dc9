"""The table build writes every entry itself: over imported tables of any
bytes it leaves the oracle's tables, twice in a row, both widths (levels of
one state up to 20 M states, boards divided into one to five regions)."""
import hashlib

import numpy as np
import pytest

import slide
from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [4, 5])
def test_build_over_imported_tables(width):
    want = load_golden("pdb_fingerprints.json")["tables"]
    with slide.Solver(width, "pdb") as s:
        rng = np.random.default_rng(width)
        for t in range(s.num_tables()):
            s.import_pdb(t, rng.integers(0, 256, s.table_size(), dtype=np.uint8))
        for _ in range(2):
            s.build_pdb()
            for t in range(s.num_tables()):
                got = hashlib.sha256(s.export_pdb(t).tobytes()).hexdigest()
                assert got == want["%d_%d" % (width, t)]["sha256"], t
