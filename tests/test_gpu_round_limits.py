"""Threshold rounds at limits no root can meet, down to the least int: nothing is
generated, and a goal among the roots is found all the same."""
import numpy as np
import pytest

import instances
import slide

pytestmark = pytest.mark.gpu

LEAST = -2 ** 31


@pytest.mark.parametrize("limit", [LEAST, LEAST + 1, LEAST + 255, LEAST + 256, -257, -256, -1])
@pytest.mark.parametrize("width,heuristic", [(4, "manhattan"), (4, "pdb"), (5, "manhattan"), (5, "pdb")])
def test_round_below_every_root(gpu_solver, width, heuristic, limit):
    s = gpu_solver(width, heuristic)
    roots = instances.random_walks(width, 8, 12, seed=3)
    roots[7] = np.arange(width * width)
    depth = np.array([0, 1, 2, 100, 200, 254, 255, 255], np.int32)
    nodes, found = s.dfs_round(roots, depth, np.full(8, -1, np.int32), limit)
    assert not np.any(nodes) and found == 255


@pytest.mark.parametrize("limit", [LEAST, LEAST + 200, -1])
@pytest.mark.parametrize("width", [4, 5])
def test_round_without_allocations_below_every_root(width, limit):
    import torch
    roots = torch.from_numpy(instances.random_walks(width, 4, 12, seed=3)).cuda()
    depth = torch.tensor([0, 1, 200, 255], dtype=torch.int32, device="cuda")
    pre = torch.full((4,), -1, dtype=torch.int32, device="cuda")
    nodes = torch.full((4,), 9, dtype=torch.int64, device="cuda")
    found = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = slide.load().sp_dfs_round_md_noalloc(width, roots.data_ptr(), depth.data_ptr(), pre.data_ptr(), 4, limit,
                                              nodes.data_ptr(), found.data_ptr(), None)
    assert st == 0
    assert not nodes.any() and int(found[0]) == -1
