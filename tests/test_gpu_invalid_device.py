"""Invalid positions in device buffers, which only the kernels see: refused,
and the next call is clean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device(engine, pos, depths):
    import torch
    d_pos = torch.from_numpy(np.ascontiguousarray(pos).view(np.int64)).cuda()
    d_out = torch.zeros(len(pos), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    engine.perft_batch_device(d_pos.data_ptr(), depths, len(pos), d_out.data_ptr())
    return [int(x) for x in d_out.cpu().numpy().view(np.uint64)]


@pytest.mark.parametrize("kings", ["none", "white", "black", "two white"])
@pytest.mark.parametrize("depth", [1, 2, 3, 4, 5, 6])
def test_positions_without_one_king_each(engine, kings, depth):
    start = engine.fen_to_pos(engine.START_FEN)
    bad = start.copy()
    bad[5] &= np.uint64({"none": 0, "white": 0xFF, "black": 0xFF << 56, "two white": 0xFFFFFFFFFFFFFFFF}[kings])
    if kings == "two white":
        bad[5] |= np.uint64(1 << 20)
        bad[0] |= np.uint64(1 << 20)
    for pos in (bad[None], np.stack([start, bad]), np.stack([bad] * 70)):
        with pytest.raises(engine.PerftError) as ei:
            _device(engine, pos, depth)
        assert ei.value.status == engine.PERFT_ERR_INVALID_ARG
    assert _device(engine, np.stack([start, start]), 3) == [8902, 8902]
    assert _device(engine, start[None], 4) == [197281]
