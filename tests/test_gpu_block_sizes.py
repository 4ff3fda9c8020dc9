"""Rounds with every block size: one block per SM, which is what a caller gets
who names none, and the blocks of 128 and 256 threads, in any number per SM."""
import pytest

import instances
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,blocks", [(256, 0), (256, 1), (256, 4), (128, 0), (128, 3)])
@pytest.mark.parametrize("width,moves", [(4, 64), (5, 74)])
def test_pdb_rounds(gpu_solver, pdb15_tables, pdb24_tables, width, moves, threads, blocks):
    states = instances.random_walks(width, 8, moves, seed=0xB5)
    want = oracle.solve(width, states, oracle.PDB, pdb15_tables if width == 4 else pdb24_tables, node_budget=3_000_000)
    pick = [i for i, w in enumerate(want) if w["len"] >= 0]
    assert pick
    s = gpu_solver(width, "pdb")
    s.set_config(threads_per_block=threads, blocks_per_sm=blocks, persistent=0)
    for i, a in zip(pick, s.solve(states[pick])):
        assert a["status"] == 0 and (a["len"], a["nodes"]) == (want[i]["len"], want[i]["nodes"]), i
