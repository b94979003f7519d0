"""The library's own choice of the select kernel (select_kernel, nbg_api.cu) on
tiles whose columns are unlike: a strip across its bounding box (occupied
columns hold fifty times the mean), density falling with distance, a thin
wall, points far apart in raw units, and ordinary ground.  It hands back few
rows (a select that does not fit hands back most), and the outputs equal the
two-pass search's bit for bit (all sum the same integers)."""
import numpy as np
import pytest

from gpupdal_b200 import abi
from gpupdal_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    rng = np.random.default_rng(17)
    if kind == "strip":
        side = 20 * np.sqrt(n)
        t, w = rng.random(n) * side, (rng.random(n) - 0.5) * 0.02 * side
        p = t + w, t - w, rng.random(n) * 40
    elif kind == "falling":
        r, a = np.exp(rng.uniform(np.log(100), np.log(10000), n)), rng.random(n) * 2 * np.pi
        p = r * np.cos(a), r * np.sin(a), rng.random(n) * 3 + r * 0.05
    elif kind == "wall":
        side = np.sqrt(n) * 20
        p = rng.random(n) * side, rng.random(n) * 8, rng.random(n) * side
    else:
        return tuple(v * np.int32(40 if kind == "far" else 1) for v in syn.stress(n, 2))
    return tuple(np.ascontiguousarray(np.round(v).astype(np.int32)) for v in p)


@pytest.mark.parametrize("kind,n,knn,most", (("strip", 200_000, 8, 0.05), ("strip", 9000, 8, 0.05),
                                             ("falling", 400_000, 8, 0.25), ("wall", 150_000, 8, 0.05),
                                             ("far", 120_000, 64, 0.0), ("far", 120_000, 32, 0.0),
                                             ("ground", 150_000, 10, 0.01)))
def test_the_librarys_choice_fits(nbg, kind, n, knn, most):
    import torch

    from gpupdal_b200.native import record_columns
    xyz = _cloud(kind, n)
    st = [abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn), abi.make_opts(abi.STAGE_NORMAL, knn=knn)]
    tile = nbg.tile(*xyz)
    tile.set_select(0)
    outs, _, stats = nbg.run(tile, st)
    tile.free()
    want = np.concatenate(outs)
    assert stats.retry_rows == 0
    tile = nbg.tile(*xyz)
    outs, _, stats = nbg.run(tile, st)
    tile.free()
    assert stats.retry_rows <= most * n
    assert np.array_equal(np.concatenate(outs), want, equal_nan=True)
    # in a batch the grid is built without its table size being read
    tile = nbg.tile(*xyz)
    rec = torch.zeros((n, 8), dtype=torch.float64, device="cuda")
    _, stats = nbg.run_batch([tile], [st], [record_columns(rec.data_ptr(), st, 64, 1)])
    torch.cuda.synchronize()
    tile.free()
    assert stats.retry_rows <= most * n
    assert np.array_equal(rec.cpu().numpy()[:, :len(want)].T, want, equal_nan=True)
