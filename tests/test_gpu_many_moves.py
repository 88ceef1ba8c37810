"""Positions with more than 218 legal moves.  No game reaches one, but the
engine accepts any placement it can search: the one-launch kernels hold 218
moves per position and hand these to the level pipeline."""
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
