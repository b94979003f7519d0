"""The group select's clump order (nbg_grid.cu) and its box tree walk
(nbg_group.cu) at the edges of clumps (32 points), blocks (1024), and levels
of the tree (32 nodes), for the neighbour counts where the list takes one, two
and three clumps of members.  Outputs equal the two-pass ring search's bit for
bit (both sum the same integers), for stage outputs and neighbour sets, and for
a subset of rows per chunk (pinned records)."""
import numpy as np
import pytest

from gpupdal_b200 import abi
from gpupdal_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _cloud(n):
    x, y, z = syn.stress(max(n, 64), 11)
    return tuple(np.ascontiguousarray(v[:n]) for v in (x, y, z))


@pytest.mark.parametrize("n", (1, 2, 31, 32, 33, 65, 97, 1023, 1024, 1025, 2049, 32769, 70001))
def test_clump_edges(nbg, n):
    x, y, z = _cloud(n)
    for knn in (3, 17, 31, 33, 49, 64):
        st = [abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn), abi.make_opts(abi.STAGE_NORMAL, knn=knn)]
        got = []
        for select in (0, 32):
            tile = nbg.tile(x, y, z)
            tile.set_select(select)
            outs, exc, _ = nbg.run(tile, st)
            ids, _ = nbg.neighbor_sets(tile, knn)
            tile.free()
            got.append((outs, np.sort(exc, order=["point_id", "stage"]), ids))
        for a, b in zip(got[0][0], got[1][0]):
            assert np.array_equal(a, b, equal_nan=True), (n, knn)
        assert np.array_equal(got[0][1], got[1][1]), (n, knn)
        assert np.array_equal(got[0][2], got[1][2]), (n, knn)


@pytest.mark.parametrize("knn,scale", ((64, 1), (40, 1), (64, 40)))
def test_long_lists_take_the_group_select(nbg, knn, scale):
    """The library's own choice for a long list (and distances past the keys'
    field: coordinates 40 times as far apart) against the two-pass search."""
    x, y, z = (v * np.int32(scale) for v in _cloud(20_000))
    st = abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn)
    ref = nbg.tile(x, y, z)
    ref.set_select(0)
    (want,), wexc, _ = nbg.run(ref, [st])
    tile = nbg.tile(x, y, z)
    (got,), exc, _ = nbg.run(tile, [st])
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.sort(exc, order="point_id"), np.sort(wexc, order="point_id"))
    tile.free()
    ref.free()


@pytest.mark.parametrize("select", (-1, 0, 2, 32))
def test_batch_select_kernels(nbg, select):
    """Tiles at the edges of the batched launches' items (128 rows, two blocks
    of 64), of every list length, against the two-pass search tile by tile."""
    import torch

    from gpupdal_b200.native import record_columns
    cases = [(n, knn) for n in (1, 63, 64, 65, 127, 129, 1025) for knn in (3, 8, 13, 17, 32)]
    cases += [(5000, 49), (20_000, 64), (20_000, 10)]
    tiles, stages, cols, recs, want = [], [], [], [], []
    for n, knn in cases:
        xyz = _cloud(n)
        st = [abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn), abi.make_opts(abi.STAGE_NORMAL, knn=knn)]
        ref = nbg.tile(*xyz)
        ref.set_select(0)
        outs, exc, _ = nbg.run(ref, st)
        ref.free()
        want.append((outs, exc))
        tile = nbg.tile(*xyz)
        if select >= 0:
            tile.set_select(select)
        rec = torch.full((n, 16), float("nan"), dtype=torch.float64, device="cuda")
        tiles.append(tile)
        stages.append(st)
        recs.append(rec)
        cols.append(record_columns(rec.data_ptr(), st, 128, 1))
    for graph in (False, True):
        for rec in recs:
            rec.fill_(float("nan"))
        got, _ = nbg.run_batch(tiles, stages, cols, graph=graph)
        torch.cuda.synchronize()
        for i, case in enumerate(cases):
            rec = recs[i].cpu().numpy()
            # rows a stage skips keep the output's previous value (NaN here, 0 in run's)
            keep = np.ones(len(rec), bool)
            keep[want[i][1]["point_id"]] = False
            for d, v in enumerate(np.concatenate(want[i][0])):
                assert np.array_equal(rec[keep, d], v[keep], equal_nan=True), (case, graph)
            key = ["point_id", "stage", "code"]
            assert np.array_equal(np.sort(got[i], order=key), np.sort(want[i][1], order=key)), (case, graph)
    for tile in tiles:
        tile.free()
