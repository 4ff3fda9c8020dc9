"""The search kernel's per-lane state at its edges: walks deeper than the
levels a lane keeps in shared memory (both block sizes keep a different
number of them), with and without donation from those levels, and tables
whose values jump over the whole byte range."""
import numpy as np
import pytest

import instances
import oracle
import slide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("lb_mode", ["none", "steal"])
@pytest.mark.parametrize("width,heuristic,moves,deep", [(4, "pdb", 80, 42), (5, "pdb", 84, 52), (4, "manhattan", 60, 30),
                                                        (5, "manhattan", 50, 30)])
def test_one_root_walked_deep(gpu_solver, pdb15_tables, pdb24_tables, width, heuristic, moves, deep, lb_mode, threads):
    tabs = (pdb15_tables if width == 4 else pdb24_tables) if heuristic == "pdb" else None
    states = instances.random_walks(width, 60, moves, seed=0xD1)
    want = oracle.solve(width, states, oracle.PDB if heuristic == "pdb" else oracle.MD, tabs, node_budget=400_000)
    picked = [i for i, w in enumerate(want) if w["len"] >= deep][:4]
    assert picked, "no instance deep enough within the budget"
    s = gpu_solver(width, heuristic)
    s.set_config(threads_per_block=threads, lb_mode=lb_mode)
    for i in picked:
        w = want[i]
        for limit, nodes in list(zip(w["f_limit"], w["nodes"]))[-2:]:
            got, found = s.dfs_round(states[i], [0], [-1], limit)
            assert int(got[0]) == nodes, (i, limit)
        assert found == w["len"]


def _tree_count(width, tiles, limit, tabs):
    """Generated nodes below one root, level by level, h from the tables."""
    n = width * width
    legal = np.array([[c // width > 0, c % width < width - 1, c % width > 0, c // width < width - 1] for c in range(n)])
    delta = np.array([-width, 1, -1, width])
    b, pre, g, count = tiles[None].copy(), np.array([-1]), 0, 0
    while len(b):
        keep = g + oracle.heuristic(width, b, oracle.PDB, tabs) <= limit
        b, pre = b[keep], pre[keep]
        blank = np.argmin(b, axis=1)
        nb, npre = [], []
        for d in range(4):
            r = np.flatnonzero(legal[blank, d] & (pre != 3 - d))
            c = b[r].copy()
            at, src = blank[r], blank[r] + delta[d]
            k = np.arange(len(r))
            c[k, at], c[k, src] = c[k, src], 0
            nb.append(c)
            npre.append(np.full(len(r), d))
        b, pre = np.concatenate(nb), np.concatenate(npre)
        count += len(b)
        g += 1
    return count


@pytest.mark.parametrize("width,limit", [(4, 24), (5, 26)])
def test_tables_of_any_bytes(width, limit):
    rng = np.random.default_rng(width)
    with slide.Solver(width, "pdb") as s:
        tabs = []
        for t in range(s.num_tables()):
            a = rng.integers(0, 7, s.table_size(), dtype=np.uint8)
            a[rng.integers(0, len(a), len(a) // 16)] = 255
            s.import_pdb(t, a)
            tabs.append(a)
        states = instances.random_permutations(width, 24, seed=5)
        h = oracle.heuristic(width, states, oracle.PDB, tabs)
        assert np.array_equal(s.heuristic_values(states), h)
        nodes, _ = s.dfs_round(states, np.zeros(24, np.int32), np.full(24, -1, np.int32), limit)
        for i, t in enumerate(states):
            assert int(nodes[i]) == _tree_count(width, t, limit, tabs), i
        assert int(nodes.max()) > 1000
