"""sp_idas_parallel at the sizes where the number of threads per root and of
roots per block changes."""
import numpy as np
import pytest

import instances
import oracle
import slide
from test_gpu_first_path import _reference_tables, _same

pytestmark = pytest.mark.gpu


def _offset(a, shift):
    """The array on the GPU at an address `shift` bytes past an allocation."""
    import torch
    flat = torch.zeros(a.size + shift, dtype=torch.uint8, device="cuda")
    flat[shift:] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1).view(np.uint8)).cuda()
    return flat


@pytest.mark.parametrize("n,moves,limit", [(1, 20, 20), (304, 14, 14), (305, 12, 14), (1024, 10, 12), (1025, 12, 12),
                                           (2047, 8, 10), (2049, 12, 10), (5000, 10, 10)])
@pytest.mark.parametrize("tables", ["none", "reference", "drifting"])
def test_every_team_size(n, moves, limit, tables):
    """The sizes where the number of threads and of roots per block changes,
    roots with and without a goal, buffers at odd addresses, and a table
    whose reverse moves do not take back what the moves added (h then depends
    on the whole walk)."""
    import torch
    roots = instances.random_walks(4, n, moves, seed=n)
    roots[::7] = instances.goal(4)
    roots[1::7] = instances.random_walks(4, len(roots[1::7]), 40, seed=n + 1)
    hd = mv = None
    if tables != "none":
        hd, mv = _reference_tables()
    if tables == "drifting":
        hd[5, 6] += 1
        hd[9, :, 2] += 1
    want = oracle.first_paths(roots, limit, hd, mv)
    shift = n % 16
    d_in = _offset(roots, shift)
    d_hd, d_mv = (None, None) if hd is None else (_offset(hd, n % 4), _offset(mv, n % 3))
    d_plan = torch.full((n, slide.SP_PLAN_STRIDE), 99, dtype=torch.int8, device="cuda")
    torch.cuda.synchronize()
    slide.idas_parallel(d_in.data_ptr() + shift, n, d_plan.data_ptr(), limit,
                        d_hd.data_ptr() + n % 4 if d_hd is not None else None,
                        d_mv.data_ptr() + n % 3 if d_mv is not None else None)
    torch.cuda.synchronize()
    got = d_plan.cpu().numpy()
    _same(got, want)
    for i in range(0, n, 97):  # nothing past the path is written
        assert np.all(got[i, 1 + max(0, int(want[i, 0])):] == 99)
