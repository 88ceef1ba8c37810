"""Positions with more than 218 legal moves.  No game reaches one, but the
engine accepts any placement it can search: the one-launch kernels hold 218
moves per position and hand these to the level pipeline."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# black to move with four king moves; after each, White has 249 moves
FEW_THEN_MANY = np.array([0xfe8181818181013f, 0x800000000000c000, 0, 0xfe8181818181017e, 0xfe8181818181013e, 0x81],
                         dtype=np.uint64)
START = 119060324  # perft(6) of the initial position


@pytest.mark.parametrize("arena", [64 << 20, 8 << 30])
def test_child_the_first_plies_kernel_cannot_hold(engine, oracle, arena):
    """k_dd_front makes the root's children; with one beyond its size the call
    is searched level by level, whatever earlier calls left in the arena."""
    assert [oracle.count(c) for c in oracle.children(FEW_THEN_MANY)] == [249] * 4
    want = {d: oracle.perft(FEW_THEN_MANY, d) for d in (5, 6)}
    start = engine.fen_to_pos(engine.START_FEN)
    try:
        engine.init(device=0, arena_bytes=arena)
        assert engine.perft(start, 6) == START  # fills the arena
        for d in (5, 6):
            for _ in range(2):  # captured, then known not to fit
                assert engine.perft(FEW_THEN_MANY, d) == want[d]
        assert engine.stats()["small_launches"] == 0
        assert engine.perft(start, 6) == START
    finally:
        engine.init(device=0, arena_bytes=8 << 30)


@pytest.mark.parametrize("n", [47, 600])
def test_levels_of_more_moves_than_the_tile_index_expects(engine, oracle, n):
    """Levels whose nodes have 249 moves each, cut at the smallest tiles
    (graph and host-driven path) and in the allocation-free entry's tiles:
    below and above the size at which the index sized for 218 would end."""
    import torch
    from perft_gpu_b200 import lib
    many = oracle.children(FEW_THEN_MANY)
    pos = np.stack([many[i % 4] for i in range(n)])
    want = np.array([oracle.perft(p, 3) for p in many], dtype=np.uint64)[np.arange(n) % 4]
    assert np.array_equal(engine.perft_batch(pos, 3), want)
    d_pos = torch.from_numpy(pos.view(np.int64)).cuda()
    d_out = torch.zeros(n, dtype=torch.int64, device="cuda")
    depths = np.full(n, 3, dtype=np.uint8)
    torch.cuda.synchronize()
    assert lib().perft_batch_noalloc(ctypes.c_void_p(d_pos.data_ptr()), ctypes.c_void_p(depths.ctypes.data),
                                     ctypes.c_uint32(n), ctypes.c_void_p(d_out.data_ptr()),
                                     ctypes.c_void_p(None)) == engine.PERFT_OK
    assert np.array_equal(d_out.cpu().numpy().view(np.uint64), want)
    engine.serve_start()
    try:
        tickets = [engine.serve_submit(p, 3) for p in pos[:100]]
        assert [engine.serve_wait(t)[0] for t in tickets] == [int(x) for x in want[:100]]
    finally:
        engine.serve_stop()
    os.environ["PERFT_NO_GRAPHS"] = "1"
    try:
        engine.init(device=0, arena_bytes=8 << 30)
        assert np.array_equal(engine.perft_batch(pos, 3), want)
    finally:
        del os.environ["PERFT_NO_GRAPHS"]
        engine.init(device=0, arena_bytes=8 << 30)
