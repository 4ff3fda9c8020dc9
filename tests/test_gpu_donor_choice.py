"""Rounds of a few roots of very different slack, so that nearly all work is
given away by size: passes of one step up, donation down to the last move and
far beyond what the lanes need, levels beyond the shared ones among them."""
import numpy as np
import pytest

import instances
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,reserve,min_slack", [(1, 0, 6), (3, 200000, 0), (33, 200000, 1)])
@pytest.mark.parametrize("width,heuristic,moves", [(4, "manhattan", 50), (4, "pdb", 70), (5, "manhattan", 46),
                                                   (5, "pdb", 84)])
def test_counts_of_uneven_roots(gpu_solver, pdb15_tables, pdb24_tables, width, heuristic, moves, steps, reserve,
                                min_slack):
    tabs = (pdb15_tables if width == 4 else pdb24_tables) if heuristic == "pdb" else None
    states = instances.random_walks(width, 16, moves, seed=0xD0)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD, tabs, node_budget=2_000_000)
    roots, nodes, cost = [], [], []
    for t, w in zip(states, want):
        for limit, n in zip(w["f_limit"], w["nodes"]):
            if w["len"] >= 0:
                roots.append(t)
                nodes.append(n)
                cost.append(limit)
    assert len(roots) >= 8 and max(nodes) > 20 * sorted(nodes)[len(nodes) // 2]
    limit = max(cost)  # one limit for all: a root's depth leaves it its own
    s = gpu_solver(width, heuristic)
    s.set_config(lb_mode="steal", steps_per_poll=steps, donate_reserve=reserve, donate_min_slack=min_slack)
    got, found = s.dfs_round(np.array(roots), limit - np.array(cost, np.int32), np.full(len(roots), -1, np.int32), limit)
    assert [int(x) for x in got] == nodes
    assert found == min(w["len"] + limit - w["f_limit"][-1] for w in want if w["len"] >= 0)
