"""The device loop publishes an iteration's roots in bulks of 32: root sets
around that size (ragged last bulk, one root, many bulks per lane), alone and
in a batch, whole threshold loops on the device."""
import pytest

import instances
import oracle
import slide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,heuristic", [(4, "manhattan"), (4, "pdb"), (5, "manhattan")])
@pytest.mark.parametrize("target", [1, 20, 32, 33, 100, 3072, 40000])
@pytest.mark.parametrize("n", [1, 7])
def test_counts_for_root_sets_around_the_bulk_size(gpu_solver, pdb15_tables, width, heuristic, target, n):
    states = instances.random_walks(width, n, 36, seed=0xB0 + n)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD,
                        pdb15_tables if heuristic == "pdb" else None)
    s = gpu_solver(width, heuristic)
    for handback in (0, 600000):
        s.set_config(frontier_target=target, handback_nodes=handback)
        got = s.solve(states)
        for i, (a, b) in enumerate(zip(got, want)):
            assert a["status"] == 0 and (a["len"], a["nodes"]) == (b["len"], b["nodes"]), (i, handback)
            assert slide.is_solution(states[i], a["moves"], width)
