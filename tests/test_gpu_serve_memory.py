"""A server whose budget is far below what its queries would take at once:
work waits for memory and every query completes with its exact count."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 24], ids=["no_table", "table"])
def server(engine, request):
    engine.init(device=0, arena_bytes=6 << 30, tt_log2_entries=request.param)
    yield engine
    engine.serve_stop()
    engine.init(device=0, arena_bytes=8 << 30)


@pytest.mark.parametrize("memory_mb", [1, 16, 32, 48, 128, 160, 320, 768, 896])
def test_small_budgets_complete(server, memory_mb):
    """Budgets at which levels with path weights, or a level and its scan,
    once took what the plies below needed."""
    pos = np.stack([server.random_playouts(seed=50 + k, n=1, min_plies=10, max_plies=26)[0] for k in range(2)] +
                   list(server.random_playouts(seed=60, n=30, min_plies=6, max_plies=30)))
    depths = np.array([7, 7] + [int(d) for d in np.random.default_rng(1).integers(3, 7, size=30)], dtype=np.uint8)
    want = [server.perft(p, int(d)) for p, d in zip(pos, depths)]
    for q in ([0], [1], range(2, 32)):  # each depth-7 query alone, then the mix
        server.serve_start(memory_bytes=memory_mb << 20)
        tickets = [server.serve_submit(pos[i], int(depths[i])) for i in q]
        deadline = time.monotonic() + 60
        while server.serve_stats()["completed"] < len(tickets) and time.monotonic() < deadline:
            time.sleep(0.002)
        st = server.serve_stats()
        assert st["completed"] == len(tickets), st
        assert [server.serve_wait(t)[0] for t in tickets] == [want[i] for i in q]
        server.serve_stop()
