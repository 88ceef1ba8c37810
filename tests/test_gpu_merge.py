"""Merged transpositions: levels from the third ply below a root on keep one
of several equal nodes, weighted by the paths that reach it."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reinit(engine, arena=8 << 30, **env):
    """Re-creates the engine under `env` and puts the environment back."""
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        engine.init(device=0, arena_bytes=arena)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


@pytest.fixture(params=["graph", "levels"])
def both_paths(engine, request):
    _reinit(engine, PERFT_DD_FORCE="1", PERFT_NO_GRAPHS="0" if request.param == "graph" else "1")
    yield engine
    engine.init(device=0, arena_bytes=8 << 30)


def _count(engine, pos, depth, memo):
    """Perft by the host move generator with remembered positions."""
    key = (pos.tobytes(), depth)
    if key not in memo:
        moves = engine.legal_moves(pos)
        memo[key] = len(moves) if depth == 1 else sum(
            _count(engine, engine.apply_move(pos, m), depth - 1, memo) for m in moves)
    return memo[key]


@pytest.mark.parametrize("depth", [5, 6, 9, 14, 18])
def test_few_pieces_deep(both_paths, depth):
    """Bare kings (and a blocked pawn pair): a few thousand positions reached
    by up to 10^12 paths each, so weights pass the narrow sums' limit (2^19)
    and 32 bits; several roots share the windows."""
    fens = ["4k3/8/8/8/8/8/8/4K3 w - - 0 1", "8/8/3k4/3p4/3P4/3K4/8/8 b - - 0 1", "k7/8/8/8/8/8/8/7K b - - 0 1"]
    pos = [both_paths.fen_to_pos(f) for f in fens]
    memo = {}
    want = [_count(both_paths, p, depth, memo) for p in pos]
    assert [both_paths.perft(p, depth) for p in pos] == want
    assert [int(x) for x in both_paths.perft_batch(np.stack(pos), depth)] == want


def test_uneven_batch(both_paths, oracle):
    """Roots of depths 1-6 in one batch: merged levels hold nodes of roots
    too shallow to merge, joining roots and equal positions of different roots."""
    pos = both_paths.random_playouts(seed=77, n=48, min_plies=0, max_plies=60)
    pos = np.concatenate([pos, pos[:16]])
    depths = (np.arange(64) % 5 + 1).astype(np.uint8)
    depths[[5, 40]] = 6
    assert np.array_equal(both_paths.perft_batch(pos, depths), oracle.perft_batch_mt(pos, depths))


def test_related_roots(engine, oracle):
    """Roots a few moves apart are searched as one tree: the children of one
    position, repeated roots, and roots that differ only in the real side to
    move; one root out of place sends the batch down the ordinary path."""
    start = engine.fen_to_pos(engine.START_FEN)
    mid = engine.random_playouts(seed=83, n=1, min_plies=16, max_plies=16)[0]
    black = start.copy()
    black[1] |= np.uint64(1 << 63)
    batches = [np.stack([engine.apply_move(p, m) for m in engine.legal_moves(p)] * k) for p, k in ((mid, 2), (start, 2))]
    batches.append(np.stack([start, black] * 16))
    batches.append(np.concatenate([batches[1], mid[None]]))
    for pos in batches:
        engine.reset_stats()
        got = engine.perft_batch(pos, 5)
        linked = engine.stats()["tt_duplicates"] > 0
        assert linked == (pos is not batches[3])
        assert np.array_equal(got, oracle.perft_batch_mt(pos, 5))


def test_fewer_items_than_paths(both_paths):
    """The count-only ply looks at each position once per root: initial
    position, depth 6, whose 197,281 four-ply paths reach 72,078 positions."""
    both_paths.reset_stats()
    start = both_paths.fen_to_pos(both_paths.START_FEN)
    assert both_paths.perft(start, 6) == 119_060_324
    assert both_paths.stats()["leaf_items"] < 4_865_609 // 2


def test_arena_without_room_for_the_set(engine, oracle):
    """Arenas down to the smallest that ran unmerged still answer."""
    start = engine.fen_to_pos(engine.START_FEN)
    try:
        for arena in (24 << 20, 6 << 20, 3 << 20):
            _reinit(engine, arena=arena, PERFT_NO_MERGE="1")
            try:
                want = engine.perft(start, 6)
            except engine.PerftError:
                want = None
            _reinit(engine, arena=arena)
            if want is not None:
                assert engine.perft(start, 6) == want == 119_060_324
    finally:
        engine.init(device=0, arena_bytes=8 << 30)


def test_served_few_pieces(engine):
    """The server's merged levels: weights beyond the narrow sums' limit, and
    queries of one level that merge next to each other."""
    fens = ["4k3/8/8/8/8/8/8/4K3 w - - 0 1", "8/8/3k4/3p4/3P4/3K4/8/8 b - - 0 1", "k7/8/8/8/8/8/8/7K b - - 0 1"]
    pos = [engine.fen_to_pos(f) for f in fens]
    memo = {}
    queries = [(p, d) for d in (6, 9, 13) for p in pos]
    engine.serve_start()
    try:
        tickets = [engine.serve_submit(p, d) for p, d in queries]
        got = [engine.serve_wait(t, timeout_s=120)[0] for t in tickets]
    finally:
        engine.serve_stop()
    assert got == [_count(engine, p, d, memo) for p, d in queries]
