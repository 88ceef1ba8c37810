"""Generation in parts and with quiet moves counted as sets (movegen.cuh,
gen_part and gen_moves_quiet), compiled for the host, against the oracle.
Runs without a GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests._oracle import P6, ROOT
from tests._positions import many_moves_with_mirrors

SRC = os.path.join(ROOT, "tests", "hostcheck", "genparts.cpp")
LIB = os.path.join(ROOT, "tests", "hostcheck", "libgenparts.so")

# en passant pinned on the rank, the file and both diagonals, evasions by it,
# double checks, castling through attack, promotions of pinned and free pawns
CRAFTED = [
    "8/8/8/K2pP2r/8/8/8/4k3 w - d6 0 1", "4k3/8/8/3pP3/8/8/8/4K3 w - d6 0 1", "4r1k1/8/8/3pP3/8/8/8/4K3 w - d6 0 1",
    "b6k/8/8/3Pp3/8/8/8/7K w - e6 0 1", "7k/8/8/4pP2/3K4/8/8/8 w - e6 0 1", "7k/6b1/8/3pP3/3K4/8/8/8 w - d6 0 1",
    "4k3/8/8/8/4r3/5n2/8/4K3 w - - 0 1", "r3k2r/8/8/8/8/8/8/R3K2R w KQkq - 0 1", "5rk1/8/8/8/8/8/8/R3K2R w KQ - 0 1",
    "1r4k1/P7/8/8/8/8/8/K7 w - - 0 1", "1b1r3k/2P5/K7/8/8/8/8/8 w - - 0 1", "2b4k/1P6/K7/8/8/8/8/8 w - - 0 1",
    "3r3k/8/8/8/8/8/3P4/3K4 w - - 0 1", "6k1/8/8/b7/8/8/3P4/4K3 w - - 0 1", "k7/8/8/8/8/8/5q2/7K w - - 0 1",
    "q5k1/8/2Q5/8/4R3/8/6B1/7K w - - 0 1",
]


@pytest.fixture(scope="module")
def gp():
    src = [SRC, os.path.join(ROOT, "perft_gpu_b200", "csrc", "tables.cpp")]
    subprocess.run(["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-o", LIB] + src, check=True)
    lib = ctypes.CDLL(LIB)
    lib.gp_replies.restype = ctypes.c_int64
    lib.gp_init()
    return lib


def _children(gp, pos):
    buf = (ctypes.c_uint64 * (6 * 256))()
    n = gp.gp_children(P6(*[int(x) for x in pos]), buf)
    assert n >= 0, n
    return sorted(tuple(buf[6 * i:6 * i + 6]) for i in range(n))


def _check_tree(gp, oracle, pos, plies):
    kids = oracle.children(pos)
    assert _children(gp, pos) == sorted(tuple(int(x) for x in k) for k in kids)
    if plies:
        for k in kids:
            _check_tree(gp, oracle, k, plies - 1)


def test_crafted_positions(gp, oracle):
    for fen in CRAFTED + list(many_moves_with_mirrors()):
        _check_tree(gp, oracle, oracle.fen_to_pos(fen), 1)


def test_playouts(gp, oracle):
    rng = np.random.default_rng(12)
    start = oracle.fen_to_pos("rnbqkbnr/pppppppp/8/8/8/8/PPPPPPPP/RNBQKBNR w KQkq - 0 1")
    for _ in range(150):
        p = start
        for _ in range(int(rng.integers(1, 120))):
            kids = oracle.children(p)
            assert _children(gp, p) == sorted(tuple(int(x) for x in k) for k in kids)
            if not len(kids):
                break
            p = kids[int(rng.integers(len(kids)))]


def _check_replies(gp, oracle, pos):
    n = ctypes.c_uint32(0)
    got = gp.gp_replies(P6(*[int(x) for x in pos]), ctypes.byref(n))
    assert got == oracle.perft(pos, 2), (oracle.pos_to_fen(pos) if hasattr(oracle, "pos_to_fen") else pos, n.value)
    return n.value


def test_quiet_replies_crafted(gp, oracle):
    """The crafted positions, two plies of each of their trees (pins, checks,
    castling rights, en passant and promotions on both sides)."""
    for fen in CRAFTED + list(many_moves_with_mirrors()):
        p = oracle.fen_to_pos(fen)
        _check_replies(gp, oracle, p)
        for k in oracle.children(p):
            _check_replies(gp, oracle, k)
            for g in oracle.children(k):
                _check_replies(gp, oracle, g)


@pytest.mark.parametrize("plies", [(0, 12), (8, 34), (40, 160)])
def test_quiet_replies_playouts(gp, oracle, plies):
    rng = np.random.default_rng(plies[1])
    start = oracle.fen_to_pos("rnbqkbnr/pppppppp/8/8/8/8/PPPPPPPP/RNBQKBNR w KQkq - 0 1")
    quiet = moves = 0
    for _ in range(200):
        p = start
        for _ in range(int(rng.integers(*plies))):
            kids = oracle.children(p)
            if not len(kids):
                break
            p = kids[int(rng.integers(len(kids)))]
            quiet += _check_replies(gp, oracle, p)
            moves += len(kids)
    assert quiet > moves // 4  # the sets do carry the bulk of the moves


@pytest.mark.parametrize("fen", [
    "4k3/8/8/8/8/8/8/B3K3 w k - 0 1", "4k2B/8/8/8/8/8/8/4K3 w k - 0 1", "B3k3/8/8/8/8/8/8/4K3 w q - 0 1",
    "4k3/8/8/8/8/8/8/4K2B w q - 0 1", "b3k3/8/8/8/8/8/8/4K3 b K - 0 1", "4k3/8/8/8/8/8/8/4K2b b K - 0 1",
    "4k2b/8/8/8/8/8/8/4K3 b Q - 0 1", "4k3/8/8/8/8/8/8/b3K3 b Q - 0 1"])
def test_quiet_replies_with_rights_that_have_no_rook(gp, oracle, fen):
    """A position's state may claim a castling right whose corner holds no
    rook; a quiet move from or to that corner takes the right all the same,
    as it does when the move is made and its replies are counted."""
    pos = oracle.fen_to_pos(fen)
    n = ctypes.c_uint32(0)
    got = gp.gp_replies(P6(*[int(x) for x in pos]), ctypes.byref(n))
    assert n.value > 0
    assert got == sum(oracle.count(np.array(k, dtype=np.uint64)) for k in _children(gp, pos))
