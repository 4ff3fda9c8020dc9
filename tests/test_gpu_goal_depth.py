"""The goal depth of a threshold round: a root's depth (0-255) plus the moves
below it, also where the sum passes 255 and the goal lies in a task that was
given away on the way."""
import numpy as np
import pytest

import instances
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [0, 200, 247, 255])
@pytest.mark.parametrize("width,heuristic,moves", [(4, "manhattan", 60), (4, "pdb", 70), (5, "manhattan", 46),
                                                   (5, "pdb", 84)])
def test_goal_depth_of_a_deep_root(gpu_solver, pdb15_tables, pdb24_tables, width, heuristic, moves, depth):
    tabs = (pdb15_tables if width == 4 else pdb24_tables) if heuristic == "pdb" else None
    states = instances.random_walks(width, 8, moves, seed=0x6D)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD, tabs, node_budget=4_000_000)
    solved = [i for i, w in enumerate(want) if w["len"] >= 0]
    at = max(solved, key=lambda i: want[i]["nodes"][-1])  # the largest tree: nearly all of it is given away
    length, count = want[at]["len"], want[at]["nodes"][-1]
    assert length > 20 and count > 1000
    s = gpu_solver(width, heuristic)
    s.set_config(lb_mode="steal", steps_per_poll=1, donate_reserve=200000, donate_min_slack=0)
    nodes, found = s.dfs_round(states[at:at + 1], [depth], [-1], depth + length)
    assert int(nodes[0]) == count
    assert found == depth + length


@pytest.mark.parametrize("width,moves", [(4, 60), (5, 46)])
def test_goal_depth_of_the_round_without_allocations(width, moves):
    import torch

    import slide
    states = instances.random_walks(width, 8, moves, seed=0x6D)
    want = oracle.solve(width, states, oracle.MD, node_budget=4_000_000)
    at = max((i for i, w in enumerate(want) if w["len"] >= 0), key=lambda i: want[i]["nodes"][-1])
    length = want[at]["len"]
    roots = torch.from_numpy(np.ascontiguousarray(states[at:at + 1])).cuda()
    depth = torch.full((1,), 255, dtype=torch.int32, device="cuda")
    pre = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    nodes = torch.zeros(1, dtype=torch.int64, device="cuda")
    found = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = slide.load().sp_dfs_round_md_noalloc(width, roots.data_ptr(), depth.data_ptr(), pre.data_ptr(), 1,
                                              255 + length, nodes.data_ptr(), found.data_ptr(), None)
    assert st == 0
    assert int(nodes[0]) == want[at]["nodes"][-1] and int(found[0]) == 255 + length
