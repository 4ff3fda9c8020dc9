"""The split pre-pass: few roots cut many levels deep (their pieces carry their
boards), goals met while splitting, both widths and heuristics."""
import pytest

import instances
import oracle
import slide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,heuristic,moves", [(4, "manhattan", 44), (4, "pdb", 60), (5, "manhattan", 44),
                                                   (5, "pdb", 70)])
@pytest.mark.parametrize("target", [1, 8, 64])
@pytest.mark.parametrize("cap", [1, 10])
def test_round_loop_with_deep_splits(gpu_solver, pdb15_tables, pdb24_tables, width, heuristic, moves, target, cap):
    tabs = (pdb15_tables if width == 4 else pdb24_tables) if heuristic == "pdb" else None
    states = instances.random_walks(width, 12, moves, seed=0x5B)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD, tabs, node_budget=3_000_000)
    pick = [i for i, w in enumerate(want) if w["len"] >= 0]
    assert pick
    s = gpu_solver(width, heuristic)
    s.set_config(persistent=0, frontier_target=target, static_split_cap=cap)
    got = s.solve(states[pick])
    for i, a in zip(pick, got):
        assert a["status"] == 0 and (a["len"], a["nodes"]) == (want[i]["len"], want[i]["nodes"]), i
        assert slide.is_solution(states[i], a["moves"], width)
