"""The one-launch grid build of small tiles (grid_small_kernel, nbg_grid.cu): at
the edges of a block (1024 points) and of its range (12288), on a plane, a strip
with more columns than it walks, a tower with more cells than it walks, and
points that all coincide, each left to the other build or built here.  The
neighbours' squared distances equal a brute-force search's (integers, exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n):
    rng = np.random.default_rng(n)
    span = {"plane": (4000, 4000, 300), "strip": (16_000_000, 1, 50), "tower": (60, 60, 16_000_000),
            "same": (1, 1, 1)}[kind]
    return [np.ascontiguousarray(rng.integers(0, s, n).astype(np.int32) - 700) for s in span]


@pytest.mark.parametrize("kind", ("plane", "strip", "tower", "same"))
@pytest.mark.parametrize("n", (1, 2, 33, 1023, 1024, 1025, 4096, 12288, 12289))
def test_neighbours_of_small_tiles(nbg, kind, n):
    import torch

    if kind == "same" and n > 1025:
        n = n % 1024 + 1025  # (every row ties with every other)
    xyz = _points(kind, n)
    p = torch.stack([torch.from_numpy(v).cuda() for v in xyz], 1).to(torch.float64)
    for knn in (3, 20):
        K = min(n, knn + 1)
        tile = nbg.tile(*xyz)
        ids, _ = nbg.neighbor_sets(tile, knn)
        tile.free()
        ids = torch.from_numpy(np.asarray(ids).astype(np.int64).reshape(n, -1)).cuda()
        assert ids.shape[1] == K
        for b in range(0, n, 2048):
            q = p[b:b + 2048]
            d = ((q[:, None, :] - p[None, :, :]) ** 2).sum(2)
            want = torch.sort(torch.topk(d, K, dim=1, largest=False).values, dim=1).values
            got = torch.sort(((p[ids[b:b + 2048]] - q[:, None, :]) ** 2).sum(2), dim=1).values
            assert torch.equal(got, want), (kind, n, knn, b)
        srt = torch.sort(ids, dim=1).values
        assert K == 1 or bool((srt[:, 1:] > srt[:, :-1]).all())
