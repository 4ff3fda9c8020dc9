"""Rounds with every block size: one block per SM, which is what a caller gets
who names none, and the blocks of 128 and 256 threads, in any number per SM."""
import pytest

import instances
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,blocks", [(256, 0), (256, 1), (256, 4), (128, 0), (128, 3)])
@pytest.mark.parametrize("width,heuristic,moves", [(4, "pdb", 64), (5, "pdb", 74), (4, "manhattan", 46),
                                                   (5, "manhattan", 44)])
def test_rounds(gpu_solver, pdb15_tables, pdb24_tables, width, heuristic, moves, threads, blocks):
    tabs = (pdb15_tables if width == 4 else pdb24_tables) if heuristic == "pdb" else None
    states = instances.random_walks(width, 8, moves, seed=0xB5)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD, tabs, node_budget=3_000_000)
    pick = [i for i, w in enumerate(want) if w["len"] >= 0]
    assert pick
    s = gpu_solver(width, heuristic)
    s.set_config(threads_per_block=threads, blocks_per_sm=blocks, persistent=0)
    for i, a in zip(pick, s.solve(states[pick])):
        assert a["status"] == 0 and (a["len"], a["nodes"]) == (want[i]["len"], want[i]["nodes"]), i
