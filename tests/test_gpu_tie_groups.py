"""Tie groups at the edge of what a warp's lanes hold (32 members): larger ones go
to the search replay, whose choice the neighbour-set export makes too.  Places
of 30 to 34 and of 70 points, with and without closer points before them; the
eigenvalues are those of the exact integer covariance of the exported sets, to
the rounding of a 3x3 solve (1e-11 of the largest)."""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knn", (8, 29, 40))
def test_groups_of_32_and_more(nbg, knn):
    rng = np.random.default_rng(8)
    pts, rows = [rng.integers(0, 3000, (2000, 3)) * (1, 1, 0) + (0, 0, 5000)], 2000
    groups = []
    for k, size in enumerate((30, 31, 32, 33, 34, 70)):
        c = np.array((10_000 + 2000 * k, 0, 0))
        # a centre with a few points near it and `size` at one place farther off
        near = c + rng.integers(-20, 21, (6, 3))
        pts += [c[None], near, np.repeat(c[None] + (100, 0, 0), size, 0), c + rng.integers(300, 900, (80, 3))]
        groups.append((rows, size))
        rows += 87 + size
    p = np.concatenate(pts).astype(np.int32)
    x, y, z = (np.ascontiguousarray(p[:, d]) for d in range(3))
    st = abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn)
    tile = nbg.tile(x, y, z)
    ids, _ = nbg.neighbor_sets(tile, knn)
    d = (p[ids.astype(np.int64)] - p[:, None, :]).astype(np.int64)
    n = ids.shape[1]
    s1 = d.sum(1)
    m = (n * np.einsum("rki,rkj->rij", d, d) - s1[:, :, None] * s1[:, None, :]) * (0.01 * 0.01) / (n * (n - 1))
    want = np.linalg.eigvalsh(m)
    ok = ~(np.abs(m) <= 1e-12).all(axis=(1, 2))
    for select in (0, 2, 32):
        tile.set_select(select)
        (got,), exc, stats = nbg.run(tile, [st])
        assert np.array_equal(np.sort(exc["point_id"]), np.flatnonzero(~ok))
        assert (np.abs(got.T[ok] - want[ok]).max(1) <= 1e-11 * want[ok, 2]).all(), select
        # the centres tie on their groups as long as these reach past the K nearest
        assert stats.tie_rows > 0 and stats.replay_rows > 0
    tile.free()
