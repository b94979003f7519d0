"""Tie rows of a tile that are many get a thread each, few a warp each
(many_ties, nbg_rows.cu).  A square lattice, where almost every row ties: the
row count on both sides of the line, through the launch whose count the device
reads, the one whose count the host knows, and the batched one.

Want: the eigenvalues of the exact integer covariance of the neighbour sets the
export gives; FP64 throughout on the device, so they agree to the rounding of a
3x3 solve, 1e-11 of the row's largest eigenvalue."""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knn", (16, 32, 63))
@pytest.mark.parametrize("w,h,sparse", ((193, 191, 0), (201, 203, 0), (203, 201, 900_000)))
def test_lattice_ties_match_their_neighbour_sets(nbg, w, h, sparse, knn):
    """36,863 and 40,803 rows; the last beside 900,000 rows that hardly tie."""
    import torch

    from gpupdal_b200.native import record_columns
    i = np.arange(w * h)
    rng = np.random.default_rng(w)
    # a lattice 5 km away from a random slab
    p = np.stack((i % w * 9, i // w * 9, np.zeros_like(i)), 1)
    p = np.concatenate((p, rng.integers((500_000, 0, 0), (900_000, 400_000, 900), (sparse, 3)))).astype(np.int32)
    x, y, z = (np.ascontiguousarray(p[:, d]) for d in range(3))
    st = abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn)
    tile = nbg.tile(x, y, z)
    ids, _ = nbg.neighbor_sets(tile, knn)
    d = (p[ids[:w * h].astype(np.int64)] - p[:w * h, None, :]).astype(np.int64)
    n = ids.shape[1]
    s1 = d.sum(1)
    m = n * np.einsum("rki,rkj->rij", d, d) - s1[:, :, None] * s1[:, None, :]
    want = np.linalg.eigvalsh(m * (0.01 * 0.01) / (n * (n - 1)))
    got = []
    for select in (0, 2, 32):
        tile.set_select(select)
        (out,), exc, stats = nbg.run(tile, [st])
        assert stats.tie_rows > 0.9 * w * h and len(exc) == 0
        got.append(out.T)
    rec = torch.zeros((len(p), 3), dtype=torch.float64, device="cuda")
    nbg.run_batch([tile], [[st]], [record_columns(rec.data_ptr(), [st], 24, 1)])
    torch.cuda.synchronize()
    got.append(rec.cpu().numpy())
    for g in got:
        err = np.abs(g[:w * h] - want).max(1)
        assert (err <= 1e-11 * want[:, 2]).all(), err.max()
        assert np.array_equal(g, got[0])
    tile.free()
