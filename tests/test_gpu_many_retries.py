"""Rows handed back by the single-pass and group selects get a thread each where
they are many, a warp each below that (many_retries, nbg_rows.cu).  Clouds that
hand every row back, on both sides of the line, alone and in a batch whose tiles
only together pass it.  All forms sum the same integers: outputs equal those of
the two-pass search, which hands no row back, bit for bit."""
import numpy as np
import pytest

from gpupdal_b200 import abi
from gpupdal_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _wall(n, seed):
    """A thin wall: a column's cells are smaller than the points' spacing."""
    rng = np.random.default_rng(seed)
    side = int(np.sqrt(n) * 20)
    return tuple(np.ascontiguousarray(rng.integers(0, s, n).astype(np.int32)) for s in (side, 8, side))


def _far(n, seed):
    """Points farther apart than the group select's keys reach."""
    return tuple(v * np.int32(40) for v in syn.stress(n, seed))


@pytest.mark.parametrize("cloud,select,knn", ((_wall, 2, 8), (_wall, 2, 13), (_far, 32, 20), (_far, 32, 64)))
@pytest.mark.parametrize("side", (-1, 1))
def test_handed_back_rows_equal_the_two_pass_search(nbg, cloud, select, knn, side):
    import torch

    from gpupdal_b200.native import record_columns
    line = 512 * torch.cuda.get_device_properties(0).multi_processor_count
    st = [abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn), abi.make_opts(abi.STAGE_NORMAL, knn=knn)]

    def run(xyz, kernel):
        tile = nbg.tile(*xyz)
        tile.set_select(kernel)
        outs, exc, stats = nbg.run(tile, st)
        tile.free()
        return np.concatenate(outs), np.sort(exc, order=["point_id", "stage"]), stats.retry_rows

    n = line + side * line // 10
    xyz = cloud(n, 3)
    want, wexc, _ = run(xyz, 0)
    got, exc, retries = run(xyz, select)
    assert (retries >= line) == (side > 0) and retries > 0.9 * n
    assert np.array_equal(got, want, equal_nan=True) and np.array_equal(exc, wexc)
    # three tiles, each below the line
    parts = [cloud(n // 3, s) for s in (4, 5, 6)]
    tiles, cols, recs = [], [], []
    for part in parts:
        tile = nbg.tile(*part)
        tile.set_select(select)
        rec = torch.zeros((n // 3, 8), dtype=torch.float64, device="cuda")
        tiles.append(tile)
        recs.append(rec)
        cols.append(record_columns(rec.data_ptr(), st, 64, 1))
    _, stats = nbg.run_batch(tiles, [st] * 3, cols)
    torch.cuda.synchronize()
    assert (stats.retry_rows >= line) == (side > 0)
    for part, tile, rec in zip(parts, tiles, recs):
        want, _, _ = run(part, 0)
        assert np.array_equal(rec.cpu().numpy()[:, :len(want)].T, want, equal_nan=True)
        tile.free()
