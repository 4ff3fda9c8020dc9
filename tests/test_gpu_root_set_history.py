"""A batch's root sets do not depend on what its solver ran before: the device
loop and the rounds have different numbers of lanes, and the cap of a large
batch's root sets goes by the rounds'."""
import pytest

import instances
import slide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,heuristic", [(4, "manhattan"), (4, "pdb"), (5, "manhattan")])
@pytest.mark.parametrize("n", [400, 500, 700])
def test_same_root_tasks_whatever_ran_last(width, heuristic, n):
    states = instances.random_walks(width, n, 30, seed=n)
    seen = []
    with slide.Solver(width, heuristic) as s:
        if heuristic == "pdb":
            s.build_pdb()
        for before in ("nothing", "device loop", "round", "rounds"):
            if before == "device loop":
                s.set_config(persistent=1, handback_nodes=0)
                s.solve(states[:3])
            elif before == "round":
                s.dfs_round(states[:3], [0] * 3, [-1] * 3, 20)
            elif before == "rounds":
                s.set_config(persistent=0)
                s.solve(states[:3])
            s.set_config(persistent=1, handback_nodes=600000)
            lens = [a["len"] for a in s.solve(states)]
            st = s.stats()
            seen.append((st["round_tasks"][0], lens))
    assert all(x == seen[0] for x in seen), [x[0] for x in seen]
