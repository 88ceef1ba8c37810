"""The index of a deep search's frontier boards (host.cpp, BoardIndex) spreads
them evenly: openings, symmetrical and open middlegames, queen endings."""
import ctypes
import os
import subprocess

import pytest

import perft_gpu_b200 as pg
from tests._oracle import P6, ROOT

SRC = os.path.join(ROOT, "tests", "hostcheck", "frontierindex.cpp")
LIB = os.path.join(ROOT, "tests", "hostcheck", "libfrontierindex.so")


@pytest.fixture(scope="module")
def fi():
    subprocess.run(["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-o", LIB, SRC,
                    os.path.join(ROOT, "perft_gpu_b200", "csrc", "tables.cpp")], check=True)
    return ctypes.CDLL(LIB)


@pytest.mark.parametrize("fen", [
    pg.START_FEN, "r3k2r/p1ppqpb1/bn2pnp1/3PN3/1p2P3/2N2Q1p/PPPBBPPP/R3K2R w KQkq - 0 1",
    "r1bq1rk1/ppp2ppp/2np1n2/2b1p3/2B1P3/2NP1N2/PPP2PPP/R1BQ1RK1 w - - 0 7", "8/2p5/3p4/KP5r/1R3p1k/8/4P1P1/8 w - - 0 1",
    "6nk/6pp/8/Q1Q1Q1Q1/8/Q1Q1Q1Q1/8/Q1Q1Q1QK w - - 0 1", "rrrrkrrr/8/8/pppppppp/PPPPPPPP/8/8/RRRRKRRR w - - 0 1"])
def test_boards_lie_near_their_first_slots(fi, fen):
    """At most half of the slots are taken, where a search for a board of a
    linear-probing table with random slots looks at 1.5 on average."""
    from tests._oracle import Oracle
    from tests.conftest import _ensure_oracle
    p = P6(*[int(x) for x in Oracle(_ensure_oracle()).fen_to_pos(fen)])
    n, probes, longest = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint64()
    for plies in (2, 3):
        assert fi.fi_probes(p, plies, ctypes.byref(n), ctypes.byref(probes), ctypes.byref(longest)) == 0
        print(fen, plies, n.value, probes.value / n.value, longest.value)
        assert probes.value <= 2 * n.value, (plies, n.value, probes.value / n.value, longest.value)
