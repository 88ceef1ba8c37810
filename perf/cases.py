"""The work that users of the engine have it do, as measurable cases.

A case is a plain dict; its "kind" names the public entry point:

  one     perft(position, depth)                     one count, host in and out
  divide  divide(position, depth)                    the subtotal of every root move
  batch   perft_batch(positions, depths)             many positions, host buffers
  device  perft_batch_device(...)                    the same on device tensors
  deep    deep(position, depth, split_plies)         host split with merged transpositions
  table   perft_batch with a transposition table     the table is cleared before each pass
  serve   serve_submit / serve_wait                  the continuous-batching server

Positions are seeded random legal playouts from the initial position, the
inputs of this repository's benchmark configurations and tests (0-40 plies,
depths 1-8).  Outputs are whole numbers (leaf counts), equal or wrong: there is
no rounding to bound, so `exact` gives no values.
"""
import math

import numpy as np
import torch

import perft_gpu_b200 as pg

# Distinct positions k plies below a playout position over its move paths of
# that length (transpositions reach a position more than once): what a search
# has to look at, whatever its order.  Sampled from 8-30-ply playouts.
DISTINCT = (1.0, 1.0, 1.0, 0.58, 0.34, 0.14, 0.08, 0.03, 0.015)
MOVES = 30.0        # mean legal moves of a playout position
OPS_COUNT = 2 * 283  # 32-bit operations to count one position's legal moves
OPS_MAKE = 2 * 41    # and to make the move that reaches it


def listed():
    return [
        # an analysis tool or a move-generator test asking for one small tree:
        # latency of a single call
        {"name": "one_d3", "kind": "one", "plies_lo": 0, "plies_hi": 40, "depth": 3},
        # perft 5 of an opening position, the size that perft suites quote
        {"name": "one_d5", "kind": "one", "plies_lo": 0, "plies_hi": 8, "depth": 5},
        # an ordinary single search of a middlegame position
        {"name": "one_d6", "kind": "one", "plies_lo": 12, "plies_hi": 28, "depth": 6},
        # a long single search of a middlegame position
        {"name": "one_d7", "kind": "one", "plies_lo": 12, "plies_hi": 28, "depth": 7},
        # the deepest plain search that a user waits for
        {"name": "opening_d8", "kind": "one", "plies_lo": 2, "plies_hi": 2, "depth": 8},
        # divided perft: the move-by-move comparison used to find generator bugs
        {"name": "divide_d6", "kind": "divide", "plies_lo": 8, "plies_hi": 30, "depth": 6},
        # a test suite's lines: a few dozen positions, shallow, host buffers
        {"name": "suite_61", "kind": "batch", "n": 61, "plies_lo": 0, "plies_hi": 40, "depth_lo": 1, "depth_hi": 4},
        # a records file's batch that is already on the device, ragged size
        {"name": "device_317", "kind": "device", "n": 317, "plies_lo": 8, "plies_hi": 30, "depth_lo": 3, "depth_hi": 5},
        # the benchmark's batch: thousands of positions of uneven depth
        {"name": "device_4096", "kind": "device", "n": 4096, "plies_lo": 8, "plies_hi": 30, "depth_lo": 4,
         "depth_hi": 6},
        # host root split of a deep search, one depth below where it pays
        {"name": "deep_d8", "kind": "deep", "plies_lo": 2, "plies_hi": 2, "depth": 8, "split": 2},
        # searches with a transposition table
        {"name": "table_d8", "kind": "table", "n": 2, "plies_lo": 12, "plies_hi": 24, "depth_lo": 8, "depth_hi": 8,
         "log2": 28},
        # a burst of queries of mixed depth through the server
        {"name": "serve_200", "kind": "serve", "n": 200, "plies_lo": 0, "plies_hi": 40, "depth_lo": 3, "depth_hi": 6},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["one", "one", "divide", "batch", "device", "device", "deep", "table", "serve"])
    lo = rng.randint(0, 24)
    case = {"kind": kind, "plies_lo": lo, "plies_hi": rng.randint(lo, 40)}
    if kind == "one":
        case["depth"] = rng.randint(2, 7)
    elif kind == "divide":
        case["depth"] = rng.randint(3, 6)
    elif kind in ("batch", "device"):
        case["depth_hi"] = rng.randint(2, 6)
        case["depth_lo"] = rng.randint(max(1, case["depth_hi"] - 3), case["depth_hi"])
        deepest = 1400 if case["depth_lo"] == 6 else 2048
        case["n"] = _log_int(rng, 2, deepest if case["depth_hi"] == 6 else 4096)
    elif kind == "deep":
        case.update(plies_lo=0, plies_hi=rng.randint(0, 3), depth=rng.randint(7, 8), split=rng.randint(1, 3))
    elif kind == "table":
        case.update(depth_lo=7, depth_hi=rng.randint(7, 8), n=rng.randint(1, 3), log2=rng.randint(24, 28),
                    plies_lo=12, plies_hi=24)
    else:
        case.update(depth_lo=rng.randint(1, 4), depth_hi=rng.randint(4, 6), n=_log_int(rng, 20, 400))
    return case


_engine = None  # the configuration of the process's engine


def _engine_for(kind, log2):
    """A user's program starts the engine (and the server) once and keeps it."""
    global _engine
    want = (kind == "serve", log2)
    if _engine == want:
        return
    pg.init(tt_log2_entries=log2)  # stops a running server
    if kind == "serve":
        pg.serve_start()
    _engine = want


def prepare(case, seed):
    kind = case["kind"]
    _engine_for(kind, case.get("log2", 0))
    n = case.get("n", 1)
    pos = pg.random_playouts(seed, n, case["plies_lo"], case["plies_hi"])
    if "depth" in case:
        depths = np.full(n, case["depth"], dtype=np.uint8)
    else:
        depths = np.random.default_rng(seed).integers(case["depth_lo"], case["depth_hi"] + 1, size=n).astype(np.uint8)
    state = {"case": case, "pos": pos, "depths": depths}
    if kind == "device":
        state["d_pos"] = torch.from_numpy(pos.view(np.int64)).cuda()
        state["d_out"] = torch.zeros(n, dtype=torch.int64, device="cuda")
    return state


def _subtotals(moves):
    """The root moves' counts in the engine's order, padded to the most moves a position has."""
    out = np.zeros(256, dtype=np.uint64)
    out[:len(moves)] = list(moves.values())
    return out


def run(state):
    case, pos, depths = state["case"], state["pos"], state["depths"]
    kind = case["kind"]
    if kind == "one":
        return pg.perft(pos[0], case["depth"])
    if kind == "divide":
        return _subtotals(pg.divide(pos[0], case["depth"]))
    if kind == "batch":
        return pg.perft_batch(pos, depths)
    if kind == "device":
        pg.perft_batch_device(state["d_pos"].data_ptr(), depths, len(depths), state["d_out"].data_ptr())
        return state["d_out"]
    if kind == "deep":
        total, moves = pg.deep(pos[0], case["depth"], case["split"])
        return {"total": total, "moves": _subtotals(moves)}
    if kind == "table":
        pg.tt_clear()
        return pg.perft_batch(pos, depths)
    tickets = [pg.serve_submit(p, int(d)) for p, d in zip(pos, depths)]
    return np.array([pg.serve_wait(t)[0] for t in tickets], dtype=np.uint64)


def work(case):
    """The distinct positions one ply above the leaves, each made and its moves
    counted once, in 32-bit integer operations; each position read and each
    count written once."""
    n = case.get("n", 1)
    lo, hi = case.get("depth_lo", case.get("depth")), case.get("depth_hi", case.get("depth"))
    counted = sum(MOVES ** (d - 1) * DISTINCT[d - 1] for d in range(lo, hi + 1)) / (hi - lo + 1)
    return {"bytes": n * (48 + 1 + 8), "flops": n * counted * (OPS_COUNT + OPS_MAKE)}


def exact(case, seed):
    return None  # whole numbers: equal or wrong
