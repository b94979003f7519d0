"""A batch of more tiles than the retry launches have rows of blocks (4 blocks a
tile fill the GPU at 592 tiles; gridDim.y ends at 65535), so that blocks take
several tiles: with few handed-back rows (warps) and with all rows handed back
(threads).  Outputs equal the two-pass search's, tile by tile."""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing,most", ((40, 0.3), (2100, 1.0)))
def test_more_tiles_than_blocks_take_at_once(nbg, spacing, most):
    import torch

    from gpupdal_b200.native import record_columns
    tiles_n, n = 640, 130
    rng = np.random.default_rng(spacing)
    st = [abi.make_opts(abi.STAGE_EIGENVALUES, knn=5)]
    side = int(spacing * np.sqrt(n))
    xyz = [tuple(np.ascontiguousarray(v) for v in
                 rng.integers(0, (side, side, spacing), (n, 3)).astype(np.int32).T) for _ in range(tiles_n)]
    for p in xyz:  # a few rows beyond the group select's reach in each tile
        p[0][:2] += 4 * side + 2300
    rec = torch.zeros((tiles_n, n, 3), dtype=torch.float64, device="cuda")
    tiles = []
    for p in xyz:
        tile = nbg.tile(*p)
        tile.set_select(32)
        tiles.append(tile)
    cols = [record_columns(rec[i].data_ptr(), st, 24, 1) for i in range(tiles_n)]
    _, stats = nbg.run_batch(tiles, [st] * tiles_n, cols, exception_capacity=16)
    torch.cuda.synchronize()
    got = rec.cpu().numpy()
    assert tiles_n <= stats.retry_rows <= most * tiles_n * n
    line = 512 * torch.cuda.get_device_properties(0).multi_processor_count
    assert (stats.retry_rows >= line) == (most == 1.0)
    for tile in tiles:
        tile.free()
    for i in range(0, tiles_n, 7):
        tile = nbg.tile(*xyz[i])
        tile.set_select(0)
        (want,), _, _ = nbg.run(tile, st)
        tile.free()
        assert np.array_equal(got[i].T, want), i
