"""The group select's first margin at the ends of its range on a tile of few
points that is 2^24 wide, where the margin's cap is far past what an int holds:
the rows whose neighbours are near are still answered, not handed back, and the
outputs equal the two-pass search's."""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("margin", (0.001, 0.5, 16.0))
def test_first_margin_on_a_wide_sparse_tile(nbg, margin):
    rng = np.random.default_rng(1)
    far = np.array([(0, 0), (16_000_000, 0), (0, 16_000_000), (16_000_000, 16_000_000)])
    xy = np.concatenate((far, 8_000_000 + rng.integers(0, 400, (67, 2))))
    xyz = (xy[:, 0], xy[:, 1], rng.integers(0, 90, len(xy)))
    x, y, z = (np.ascontiguousarray(v).astype(np.int32) for v in xyz)
    st = abi.make_opts(abi.STAGE_EIGENVALUES, knn=64)
    got = []
    for select in (0, 32):
        tile = nbg.tile(x, y, z)
        tile.set_select(select, margin)
        (out,), exc, stats = nbg.run(tile, [st])
        tile.free()
        assert len(exc) == 0 and stats.retry_rows <= (8 if select else 0)
        got.append(out)
    assert np.array_equal(got[0], got[1])
