"""Batches of small trees in one launch (k_small_trees)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 63, 64, 65])
@pytest.mark.parametrize("depths", [(0, 4), (4, 4), (1, 3), (0, 0)])
def test_small_batches_equal_oracle(engine, oracle, n, depths):
    """Sizes around the largest batch of the one-launch kernel, depths 0-4,
    host and device buffers."""
    import torch
    pos = engine.random_playouts(seed=300 + n, n=n, min_plies=0, max_plies=90)
    d = np.random.default_rng(n).integers(depths[0], depths[1] + 1, size=n).astype(np.uint8)
    want = oracle.perft_batch_mt(pos, d)
    assert np.array_equal(engine.perft_batch(pos, d), want)
    d_pos = torch.from_numpy(pos.view(np.int64)).cuda()
    d_out = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        engine.perft_batch_device(d_pos.data_ptr(), d, n, d_out.data_ptr())
        assert np.array_equal(d_out.cpu().numpy().view(np.uint64), want)


def test_positions_the_kernel_cannot_hold(engine, oracle):
    """A position with more pieces than move groups (and one with more moves
    than any game's) goes to the level pipeline, alone and in a batch; an
    invalid one is refused, and the next call is clean."""
    queens = engine.fen_to_pos("QQQQQQQQ/QQQQQQQQ/QQQQQQQQ/8/8/8/7p/K6k b - - 0 1")
    many = engine.fen_to_pos("3Q4/1Q4Q1/4Q3/2Q4R/Q4Q2/3Q4/1Q4Rp/1K1BBNNk w - - 0 1")  # 218 moves
    start = engine.fen_to_pos(engine.START_FEN)
    pos = np.stack([start, queens, many])
    for d in (2, 3):
        want = [oracle.perft(p, d) for p in pos]
        assert [engine.perft(p, d) for p in pos] == want
        assert [int(x) for x in engine.perft_batch(pos, d)] == want
    bad = start.copy()
    bad[5] = 0
    with pytest.raises(engine.PerftError) as ei:
        engine.perft_batch(np.stack([start, bad]), 3)
    assert ei.value.status == engine.PERFT_ERR_INVALID_ARG
    assert [int(x) for x in engine.perft_batch(np.stack([start, start]), 3)] == [8902, 8902]


def test_first_two_plies_in_one_launch(engine, oracle):
    """Single roots below depth 5 start from the second ply (k_dd_front): a
    mated and a stalemated root, a root whose moves all mate or stalemate,
    bare kings, and playouts of every phase."""
    fens = ["rnb1kbnr/pppp1ppp/8/4p3/6Pq/5P2/PPPPP2P/RNBQKBNR w KQkq - 0 1", "7k/5Q2/6K1/8/8/8/8/8 b - - 0 1",
            "7k/8/5QK1/8/8/8/8/8 b - - 0 1", "4k3/8/8/8/8/8/8/4K3 w - - 0 1"]
    pos = [engine.fen_to_pos(f) for f in fens]
    pos += list(engine.random_playouts(seed=611, n=4, min_plies=0, max_plies=6))
    pos += list(engine.random_playouts(seed=612, n=8, min_plies=60, max_plies=200))
    for p in pos:
        assert engine.perft(p, 6) == oracle.perft(p, 6)


def test_small_batches_and_level_graphs_are_told_apart(engine, oracle, monkeypatch):
    """A batch in one launch is one graph launch without a count-only or
    interior launch; with the one-launch kernel off, batches of the same
    depths are captured and replayed as graphs of levels."""
    pos = engine.random_playouts(seed=71, n=32, min_plies=2, max_plies=40)
    want = {d: oracle.perft_batch_mt(pos, d) for d in (2, 3, 4)}
    try:
        for small in ("1", "0"):
            monkeypatch.setenv("PERFT_SMALL_TREE", small)
            engine.init(device=0, arena_bytes=4 << 30)
            engine.reset_stats()
            for _ in range(3):  # with levels: captured, then replayed
                for d in (2, 3, 4):
                    assert np.array_equal(engine.perft_batch(pos, d), want[d])
            st = engine.stats()
            assert st["graph_launches"] == 9 and st["small_launches"] == 0
            if small == "1":
                assert st["leaf_launches"] == st["expand_launches"] == st["leaf_items"] == 0
                assert st["other_launches"] == 9
            else:
                assert st["leaf_launches"] == 9 and st["expand_launches"] == 9
                assert st["leaf_items"] > 0 and st["leaf_parents"] > 0 and st["leaf_ms"] > 0
    finally:
        monkeypatch.delenv("PERFT_SMALL_TREE")
        engine.init(device=0, arena_bytes=8 << 30)


def test_more_moves_than_the_kernel_holds(engine, oracle):
    """Positions with 249 moves as a root and as the children of a root with
    four moves: counted by the level pipeline, alone and in a batch."""
    few = np.array([0xfe8181818181013f, 0x800000000000c000, 0, 0xfe8181818181017e, 0xfe8181818181013e, 0x81],
                   dtype=np.uint64)
    many = oracle.children(few)[0]
    assert oracle.count(few) == 4 and oracle.count(many) == 249
    above = engine.random_playouts(seed=5, n=1, min_plies=8, max_plies=8)[0]
    for p, depths in ((many, (2, 3, 4)), (few, (3, 4, 5))):
        for d in depths:
            want = oracle.perft(p, d)
            engine.reset_stats()
            assert engine.perft(p, d) == want
            assert engine.stats()["small_launches"] == 0
            if d <= 4:
                engine.reset_stats()
                assert [int(x) for x in engine.perft_batch(np.stack([above, p, p]), d)] == \
                    [oracle.perft(above, d), want, want]
                assert engine.stats()["leaf_launches"] > 0
    assert engine.perft(above, 4) == oracle.perft(above, 4)
