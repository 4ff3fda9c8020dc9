"""Performance cases of the framework: the calls that its users make, at the
sizes they make them.

  solve    a batch of instances to optimal answers (sp_solve_batch, or
           sp_solve_batch_device when the tiles already are on the GPU)
  start    a program from nothing to its first answers: create a solver, build
           the pattern databases, solve a few instances, close it
  label    one threshold round over a caller's roots from host memory, with
           the roots' heuristic values first: how the balancer's training
           tuples are labelled (train_lb.label), and the call that stands in
           for the reference's dfs_kernel
  round    the same threshold round on device buffers without any allocation
           (sp_dfs_round_md_noalloc)
  gradient one forward and backward pass of the learned balancer's model
  predict  its inference on host rows
  first    the first-path search of every root on its own (sp_idas_parallel)

Searches return whole numbers only (lengths, thresholds, node counts).  The
move sequence is left out: every goal of the last threshold is an optimal
answer, and which one is met first is not fixed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sliding-puzzle_gb300"))

import instances  # noqa: E402
import slide  # noqa: E402
import train_lb  # noqa: E402

HIDDEN = 256  # the model's hidden width (both layers)


def listed():
    return [
        # one easy 15-puzzle: the smallest call, all latency and launches
        {"name": "solve15_md_walk40_1", "kind": "solve", "width": 4, "heuristic": "manhattan", "source": "walk40",
         "n": 1, "device": False},
        # one random 15-puzzle with pattern databases: an interactive call
        {"name": "solve15_pdb_random_1", "kind": "solve", "width": 4, "heuristic": "pdb", "source": "random",
         "n": 1, "device": False},
        # the headline workload: 100 random 15-puzzles, tiles in device memory
        {"name": "solve15_pdb_random_100", "kind": "solve", "width": 4, "heuristic": "pdb", "source": "random",
         "n": 100, "device": True},
        # bulk solving: half walks of 40-80 moves, half random permutations
        {"name": "solve15_pdb_mixed_4096", "kind": "solve", "width": 4, "heuristic": "pdb", "source": "mixed",
         "n": 4096, "device": False},
        # 100 walks of 60 moves without tables
        {"name": "solve15_md_walk60_100", "kind": "solve", "width": 4, "heuristic": "manhattan", "source": "walk60",
         "n": 100, "device": False},
        # the reference's own 24-puzzle set: 50 instances of its generator
        {"name": "solve24_pdb_reference_50", "kind": "solve", "width": 5, "heuristic": "pdb", "source": "reference",
         "n": 50, "device": False},
        # a 24-puzzle program that starts cold (the tables are not shipped)
        {"name": "start24_pdb_8", "kind": "start", "width": 5, "n": 8},
        # a labelling chunk of the learned balancer's training set
        {"name": "label24_16384", "kind": "label", "width": 5, "heuristic": "pdb", "n": 16384, "slack": 4},
        # a threshold round over a root set of the reference's BLOCK_NUM
        {"name": "round24_md_2048", "kind": "round", "width": 5, "n": 2048, "slack": 4},
        # a training batch of the balancer's model (train_lb's default)
        {"name": "gradient24_8192", "kind": "gradient", "width": 5, "n": 8192},
        # predictions for a root set
        {"name": "predict24_60000", "kind": "predict", "width": 5, "n": 60000},
        # a root set searched root by root, paths back
        {"name": "first15_4096", "kind": "first", "n": 4096, "moves": 26},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["solve15pdb", "solve15md", "solve24pdb", "solve24md", "start", "label", "round", "gradient",
                       "predict", "first"])
    if kind == "solve15pdb":
        return {"kind": "solve", "width": 4, "heuristic": "pdb", "source": rng.choice(["random", "mixed"]),
                "n": _log_int(rng, 2, 1200), "device": rng.random() < 0.5}
    if kind == "solve15md":
        return {"kind": "solve", "width": 4, "heuristic": "manhattan", "source": "walk%d" % rng.randint(30, 60),
                "n": _log_int(rng, 1, 600), "device": rng.random() < 0.5}
    if kind == "solve24pdb":
        return {"kind": "solve", "width": 5, "heuristic": "pdb",
                "source": rng.choice(["reference", "walk%d" % rng.randint(50, 90)]), "n": _log_int(rng, 1, 80),
                "device": rng.random() < 0.5}
    if kind == "solve24md":
        return {"kind": "solve", "width": 5, "heuristic": "manhattan", "source": "walk%d" % rng.randint(24, 46),
                "n": _log_int(rng, 1, 150), "device": rng.random() < 0.5}
    if kind == "start":
        return {"kind": "start", "width": 4, "n": _log_int(rng, 1, 60)}
    if kind == "label":
        return {"kind": "label", "width": rng.choice([4, 5]), "heuristic": rng.choice(["pdb", "manhattan"]),
                "n": _log_int(rng, 200, 16000), "slack": rng.randint(1, 4)}
    if kind == "round":
        return {"kind": "round", "width": rng.choice([4, 5]), "n": _log_int(rng, 100, 16000),
                "slack": rng.randint(1, 4)}
    if kind == "gradient":
        return {"kind": "gradient", "width": rng.choice([4, 5]), "n": 128 * _log_int(rng, 1, 250)}
    if kind == "predict":
        return {"kind": "predict", "width": rng.choice([4, 5]), "n": _log_int(rng, 100, 60000)}
    return {"kind": "first", "n": _log_int(rng, 30, 6000), "moves": rng.randint(16, 26)}


@functools.lru_cache(maxsize=None)
def _solver(width, heuristic):
    """The solver that a program keeps for all its calls."""
    s = slide.Solver(width, heuristic)
    if heuristic == "pdb":
        s.build_pdb()
    return s


def _tiles(width, source, n, seed):
    if source == "random":
        return instances.random_permutations(width, n, seed)
    if source == "mixed":
        a = (n + 1) // 2
        return np.concatenate([instances.random_walks(width, a, (40, 80), seed),
                               instances.random_permutations(width, n - a, seed + 1)])
    if source == "reference":
        return instances.reference_walks(width, n, seed)
    return instances.random_walks(width, n, int(source[4:]), seed)


def _slacks(n, most, seed):
    return np.random.default_rng(seed).integers(0, most + 1, n).astype(np.int32)


def _manhattan(tiles, width):
    t = tiles.astype(np.int64)
    c = np.arange(width * width)
    d = np.abs(t // width - c // width) + np.abs(t % width - c % width)
    return np.where(t > 0, d, 0).sum(axis=1)


def _walk_range(width):
    """Walk lengths of the balancer's training states (train_lb)."""
    return (100, 220) if width == 5 else (40, 80)


def _model(width, seed):
    """Weights as a trained model's order of magnitude: He-normal layers and
    the mean log2 size as the last bias."""
    rng = np.random.default_rng(seed)
    tiles = width * width
    rows = (tiles - 1) * tiles + 1
    return np.concatenate([
        rng.normal(0, math.sqrt(2.0 / tiles), rows * HIDDEN), np.zeros(HIDDEN),
        rng.normal(0, math.sqrt(2.0 / HIDDEN), HIDDEN * HIDDEN), np.zeros(HIDDEN),
        rng.normal(0, math.sqrt(1.0 / HIDDEN), HIDDEN), [8.0]]).astype(np.float32)


def _model_inputs(case, seed):
    width, n = case["width"], case["n"]
    tiles = train_lb.vector_walks(width, n, *_walk_range(width), seed)
    slack = _slacks(n, 7, seed + 1)
    noise = np.random.default_rng(seed + 2).normal(0, 2, n)
    target = np.maximum(0, 3.0 * slack + 2 + noise).astype(np.float32)
    return _model(width, seed + 3), tiles, slack, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        tiles = _tiles(case["width"], case["source"], case["n"], seed)
        s = {"kind": kind, "solver": _solver(case["width"], case["heuristic"]), "tiles": tiles}
        if case["device"]:
            s["device"] = torch.from_numpy(tiles).cuda()
            torch.cuda.synchronize()
        return s
    if kind == "start":
        slide.load()
        return {"kind": kind, "width": case["width"], "tiles": _tiles(case["width"], "walk60", case["n"], seed)}
    if kind in ("label", "round"):
        width, n = case["width"], case["n"]
        tiles = train_lb.vector_walks(width, n, *_walk_range(width), seed)
        slack = _slacks(n, case["slack"], seed + 1)
        if kind == "label":
            return {"kind": kind, "solver": _solver(width, case["heuristic"]), "tiles": tiles, "slack": slack}
        h = _manhattan(tiles, width)
        limit = int((h + 2 * slack).max())
        return {"kind": kind, "width": width, "n": n, "limit": limit, "lib": slide.load(),
                "roots": torch.from_numpy(tiles).cuda(),
                "depth": torch.from_numpy((limit - h - 2 * slack).astype(np.int32)).cuda(),
                "pre": torch.full((n,), -1, dtype=torch.int32, device="cuda"),
                "nodes": torch.zeros(n, dtype=torch.int64, device="cuda"),
                "found": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if kind in ("gradient", "predict"):
        weights, tiles, slack, target = _model_inputs(case, seed)
        solver = slide.Solver(case["width"], "manhattan")
        solver.lbm_import(weights)
        return {"kind": kind, "solver": solver, "tiles": tiles, "slack": slack, "target": target}
    roots = train_lb.vector_walks(4, case["n"], case["moves"], case["moves"], seed)
    return {"kind": kind, "n": case["n"], "limit": case["moves"], "roots": torch.from_numpy(roots).cuda(),
            "plan": torch.zeros(case["n"], slide.SP_PLAN_STRIDE, dtype=torch.int8, device="cuda")}


_RESULT = np.dtype(slide.SpResult)


def _answers(raw, n):
    r = np.frombuffer(raw, dtype=_RESULT)[:n]
    return {k: r[k] for k in ("status", "len", "n_iter", "f_limit", "nodes")}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        n = state["tiles"].shape[0]
        if "device" in state:
            return _answers(state["solver"].solve_device_raw(state["device"].data_ptr(), n), n)
        return _answers(state["solver"].solve_raw(state["tiles"]), n)
    if kind == "start":
        with slide.Solver(state["width"], "pdb") as solver:
            solver.build_pdb()
            return _answers(solver.solve_raw(state["tiles"]), state["tiles"].shape[0])
    if kind == "label":
        solver = state["solver"]
        h = solver.heuristic_values(state["tiles"])
        cost = h + 2 * state["slack"]
        limit = int(cost.max())
        nodes, found = solver.dfs_round(state["tiles"], limit - cost, np.full(len(h), -1, np.int32), limit)
        return {"h": h, "nodes": nodes.view(np.int64), "found": found}
    if kind == "round":
        s = state
        st = s["lib"].sp_dfs_round_md_noalloc(s["width"], s["roots"].data_ptr(), s["depth"].data_ptr(),
                                              s["pre"].data_ptr(), s["n"], s["limit"], s["nodes"].data_ptr(),
                                              s["found"].data_ptr(), None)
        return {"status": st, "nodes": s["nodes"], "found": s["found"]}
    if kind == "gradient":
        loss, grads = state["solver"].lbm_gradients(state["tiles"], state["slack"], state["target"])
        return {"loss": loss, "grads": grads}
    if kind == "predict":
        return state["solver"].lbm_predict(state["tiles"], state["slack"])
    slide.idas_parallel(state["roots"].data_ptr(), state["n"], state["plan"].data_ptr(), state["limit"])
    return state["plan"]


# Mean generated nodes per instance (measured; the spread between batches is
# large): walks by their length, whole sets as they are.
_MEAN_NODES = {
    (4, "manhattan"): {24: 5e3, 30: 1.6e4, 40: 4e5, 50: 2.8e6, 60: 9e6},
    (5, "manhattan"): {24: 5e3, 30: 3e4, 40: 2e5, 50: 5e6},
    (4, "pdb"): {"random": 1.2e7, "mixed": 6e6, 60: 1e6},
    (5, "pdb"): {"reference": 5e6, 50: 3e5, 60: 9e5, 80: 7e6, 100: 3e7},
}
# Mean generated nodes per root of a threshold round, by slack in steps of two
_ROUND_GROWTH = {(4, "manhattan"): 5.0, (5, "manhattan"): 8.0, (4, "pdb"): 7.0, (5, "pdb"): 11.0}


def _mean_nodes(width, heuristic, source):
    t = _MEAN_NODES[width, heuristic]
    if source in t:
        return t[source]
    m = int(source[4:])
    at = sorted(k for k in t if isinstance(k, int))
    return math.exp(np.interp(m, at, [math.log(t[k]) for k in at]))


def _search_work(nodes, heuristic):
    """A generated node costs one regular and one reflected table sector, or
    the integer operations of the serial Manhattan search."""
    if heuristic == "pdb":
        return {"bytes": nodes * slide.PDB_BYTES_PER_NODE, "flops": 0}
    return {"bytes": 0, "flops": nodes * slide.MD_OPS_PER_NODE}


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "solve":
        return _search_work(n * _mean_nodes(case["width"], case["heuristic"], case["source"]), case["heuristic"])
    if kind == "start":
        # every table entry is written once
        w = _search_work(n * _mean_nodes(case["width"], "pdb", "walk60"), "pdb")
        return {"bytes": w["bytes"] + slide.pdb_table_bytes(case["width"]), "flops": 0}
    if kind in ("label", "round"):
        heuristic = case.get("heuristic", "manhattan")
        g, s = _ROUND_GROWTH[case["width"], heuristic], case["slack"]
        return _search_work(n * 20.0 * (g ** (s + 1) - 1) / (g - 1) / (s + 1), heuristic)
    if kind in ("gradient", "predict"):
        tiles = case["width"] ** 2
        rows = (tiles - 1) * tiles + 1
        params = rows * HIDDEN + HIDDEN * HIDDEN + 3 * HIDDEN + 1
        per_row = 2 * HIDDEN * HIDDEN + 2 * tiles * HIDDEN  # layer 2, and layer 1 as a gather-sum
        if kind == "predict":
            return {"bytes": n * (tiles + 8) + 4 * params, "flops": n * per_row}
        return {"bytes": n * (tiles + 8) + 8 * params, "flops": 3 * n * per_row}
    # first: a root's tiles in, its plan row out, and a serial walk in between
    return {"bytes": n * (16 + slide.SP_PLAN_STRIDE),
            "flops": n * slide.MD_OPS_PER_NODE * 1.3 ** (case["moves"] - 4)}


def exact(case, seed):
    """The model's loss, gradients and predictions in 64 bits; searches
    return whole numbers only."""
    if case["kind"] not in ("gradient", "predict"):
        return None
    weights, tiles, slack, target = _model_inputs(case, seed)
    cells = case["width"] ** 2
    rows = (cells - 1) * cells + 1
    n = len(tiles)
    sizes = [rows * HIDDEN, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN, 1]
    w1, b1, w2, b2, w3, b3 = torch.from_numpy(weights).double().split(sizes)
    w1, w2 = w1.view(rows, HIDDEN), w2.view(HIDDEN, HIDDEN)
    place = torch.from_numpy(np.argsort(tiles.astype(np.int64), axis=1)[:, 1:].copy())  # cell of each tile
    x = torch.zeros(n, rows, dtype=torch.float64)
    x.scatter_(1, place + torch.arange(cells - 1) * cells, 1.0)
    x[:, -1] = torch.from_numpy(slack).double()
    z1 = x @ w1 + b1
    h1 = z1.clamp(min=0)
    z2 = h1 @ w2.T + b2
    h2 = z2.clamp(min=0)
    y = h2 @ w3 + b3
    if case["kind"] == "predict":
        return y
    off = y - torch.from_numpy(target).double()
    dy = 2 * off / n
    d2 = dy[:, None] * w3 * (z2 > 0)
    d1 = d2 @ w2 * (z1 > 0)
    grads = torch.cat([(x.T @ d1).flatten(), d1.sum(0), (d2.T @ h1).flatten(), d2.sum(0), h2.T @ dy, dy.sum()[None]])
    return {"loss": (off * off).mean().item(), "grads": grads}
