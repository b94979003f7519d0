"""Rows answered by whole warps (nbg_rows.cu): tie rows and the rows the
single-pass select hands back, at the neighbour counts where the list held
across the lanes takes one, two and three registers.

Want: the eigenvalues of the exact covariance of the neighbour sets that the
neighbour-set export gives (one thread per row, its own tie order).  The
device's eigenvalues come from the same integers with FP64 arithmetic
throughout, so they agree to FP64 rounding of a 3x3 solve: 1e-11 of the row's
largest eigenvalue.  (Members of a tie group at one FP64 distance with one
offset are interchangeable in the sums; with distinct offsets both paths order
them on the same tree.)
"""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


def _clouds():
    rng = np.random.default_rng(5)
    # a lattice: groups of 6, 8, 12 and 24 at one distance, in sets of any size
    g = np.arange(12, dtype=np.int32) * 9
    lat = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    # clumps, a sparse halo around them (long ring searches) and duplicates
    c = rng.integers(0, 4000, (12, 3))
    clump = (c[rng.integers(0, 12, 3000)] + rng.normal(0, 25, (3000, 3))).astype(np.int32)
    halo = rng.integers(-1500, 5500, (150, 3)).astype(np.int32)
    pts = np.concatenate((clump, halo, clump[:400], clump[:30], clump[:30]))
    # 45 points at one place: a tie group past the lanes goes to the search replay
    pts = np.concatenate((pts, np.repeat(clump[:1], 45, axis=0)))
    return {"lattice": lat, "clumps": pts[rng.permutation(len(pts))]}


@pytest.mark.parametrize("knn", (1, 8, 30, 31, 32, 62, 63, 64))
@pytest.mark.parametrize("name", ("lattice", "clumps"))
def test_warp_rows_match_their_neighbour_sets(nbg, name, knn):
    p = _clouds()[name].astype(np.int32)
    x, y, z = (np.ascontiguousarray(p[:, d]) for d in range(3))
    st = abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn)
    tile = nbg.tile(x, y, z)
    ids, _ = nbg.neighbor_sets(tile, knn)
    d = (p[ids.astype(np.int64)] - p[:, None, :]).astype(np.int64)
    n = ids.shape[1]
    s1 = d.sum(1)
    m = n * np.einsum("rki,rkj->rij", d, d) - s1[:, :, None] * s1[:, None, :]
    want = np.linalg.eigvalsh(m * (0.01 * 0.01) / (n * (n - 1)))
    skipped = (np.abs(m * (0.01 * 0.01) / (n * (n - 1))) <= 1e-12).all(axis=(1, 2))
    handed = 0
    for select in (0, 2):
        tile.set_select(select)
        (got,), exc, stats = nbg.run(tile, [st])
        handed += stats.retry_rows
        assert stats.tie_rows > 0
        assert np.array_equal(np.sort(exc["point_id"]), np.flatnonzero(skipped))
        ok = ~skipped
        err = np.abs(got.T[ok] - want[ok]).max(1)
        assert (err <= 1e-11 * want[ok, 2]).all(), f"select {select}: {err.max():.2e}"
    assert handed > 0 or name == "lattice"
    tile.free()
