"""The count-only ply compares the moves it generates for a counted parent
with the count, as interior plies do (movegen.cuh, moves_as_counted),
compiled for the host.  Runs without a GPU."""
import ctypes
import os
import re
import subprocess

from tests._oracle import P6, ROOT

SRC = os.path.join(ROOT, "tests", "hostcheck", "leafcheck.cpp")
LIB = os.path.join(ROOT, "tests", "hostcheck", "libleafcheck.so")
CSRC = os.path.join(ROOT, "perft_gpu_b200", "csrc")


def test_generated_moves_are_compared_with_the_count(oracle):
    subprocess.run(["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-o", LIB, SRC, os.path.join(CSRC, "tables.cpp")],
                   check=True)
    lib = ctypes.CDLL(LIB)
    lib.lc_init()
    p = oracle.fen_to_pos("r3k2r/p1ppqpb1/bn2pnp1/3PN3/1p2P3/2N2Q1p/PPPBBPPP/R3K2R w KQkq - 0 1")
    for _ in range(40):
        kids = oracle.children(p)
        pos, n = P6(*[int(x) for x in p]), len(kids)
        if n < 3:
            break
        assert lib.lc_agrees(pos, n, 0)
        # a generator that lost or repeated a move, against the oracle's count
        assert not lib.lc_agrees(pos, n, 1) and not lib.lc_agrees(pos, n, -1)
        assert lib.lc_agrees(pos, 1, 0)  # not counted
        p = kids[n // 2]


def test_the_kernel_raises_the_error():
    src = open(os.path.join(CSRC, "engine.cu")).read()
    leaf = src[src.index(" k_leaf(const TileParams"):]
    leaf = leaf[:leaf.index("\n}\n")]
    assert re.search(r"!moves_as_counted\([^;]*\)\s*\)\s*atomicOr\(P\.err, DERR_GEN_MISMATCH\);", leaf)
