"""The counting form of the radius kernel (radius outliers) at the edges of its
blocks and of min_k, against a brute-force count: at a radius whose square lies
between two integers (raw units) the count is exact."""
import numpy as np
import pytest

from gpupdal_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1, 2, 127, 128, 129, 3000))
def test_counts_equal_brute_force(nbg, n):
    rng = np.random.default_rng(n)
    xyz = [np.ascontiguousarray(rng.integers(-300, s, n).astype(np.int32)) for s in (900, 900, -100)]
    p = np.stack(xyz, 1).astype(np.int64)
    cnt = np.concatenate([(((q[:, None] - p[None]) ** 2).sum(2) < 2550.25).sum(1)
                          for q in np.array_split(p, max(1, n // 500))])
    for min_k in (0, 1, 2, 7, 1000):
        tile = nbg.tile(*xyz)
        _, _, stats = nbg.run(tile, [abi.consumer_opts(abi.STAGE_OUTLIER, method="radius", radius=0.505,
                                                       min_k=min_k)])
        tile.free()
        assert stats.inliers == int((cnt > min_k).sum()), (n, min_k)
        assert stats.outliers == n - int((cnt > min_k).sum()), (n, min_k)
