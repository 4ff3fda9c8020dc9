"""A solver whose first call is a threshold round (or the stall self-test) has
room for a batch afterwards: the device loop keeps two limits and two solution
records per instance."""
import pytest

import instances
import oracle
import slide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["round", "selftest"])
@pytest.mark.parametrize("n", [33, 64, 65])
def test_batch_after_a_first_round(first, n):
    states = instances.random_walks(4, n, 20, seed=n)
    with slide.Solver(4, "manhattan") as s:
        if first == "round":
            s.dfs_round(states[:1], [0], [-1], 20)
        else:
            assert s.selftest_stall(200) == -8
        got = s.solve(states)
        want = oracle.solve(4, states, oracle.MD)
        for a, b in zip(got, want):
            assert a["status"] == 0 and (a["len"], a["nodes"]) == (b["len"], b["nodes"])
