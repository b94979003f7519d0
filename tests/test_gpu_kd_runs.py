"""The KD replica where a segment's split falls among points at its cut (odd
columns of a raster, coincident points), at the level passes (segments above
4096 points): runs read by one warp and by all, several a level, in short and
long tiles; and trees of uneven leaves,
one of them past the room that the nodes get at first
(of those the point order is compared).  The exported tree equals the
oracle's."""
import numpy as np
import pytest

from . import _util as U

pytestmark = pytest.mark.gpu


def _raster(w, h, step=50, flat=False):
    i = np.arange(w * h)
    x, y = i % w * step, i // w * step
    return x, y, np.zeros_like(i) if flat else (200 * np.sin(x / 900.0) * np.cos(y / 700.0)).astype(np.int64)


def _cloud(kind):
    rng = np.random.default_rng(4)
    if kind == "coincident":  # one run of all points, level after level
        return np.full(30_000, 7), np.full(30_000, -3), np.full(30_000, 12)
    if kind == "stack":  # a run above 4096 points in a cloud, with other coordinates spread
        n = 20_000
        return np.where(rng.random(n) < 0.5, 500, rng.integers(0, 1001, n)), rng.integers(0, 400, n), rng.integers(0, 60, n)
    if kind == "columns":  # few distinct x: long runs with every point of a column
        n = 60_000
        return rng.integers(0, 9, n) * 2000, rng.integers(0, 3000, n), rng.integers(0, 500, n)
    if kind == "nested":  # clusters inside clusters: leaves of few points
        s = np.exp(rng.uniform(0, np.log(8e6), 50_000))
        d = rng.normal(size=(3, 50_000))
        return tuple(np.round(d / np.linalg.norm(d, axis=0) * s))
    if kind.startswith("peeled"):  # places whose splits take off one point at a time
        places, bits, pile = (1024, 14, 101) if kind == "peeled" else (2048, 13, 88)
        arms = [np.eye(3, dtype=np.int64)[d] << k for d in range(3) for k in range(1, bits - 1 if d == 0 else 23)]
        one = np.concatenate((arms, np.zeros((pile, 3), np.int64)))
        at = np.arange(places)[:, None] * np.array((1 << bits, 0, 0))
        return tuple((at[:, None] + one[None]).reshape(-1, 3).T)
    w, h, flat = {"raster": (101, 99, False), "flat": (201, 203, True), "wide": (601, 401, False),
                  "long tiles": (1801, 1601, False)}[kind]
    return _raster(w, h, flat=flat)


@pytest.mark.parametrize("kind", ("raster", "flat", "wide", "long tiles", "coincident", "stack", "columns", "nested", "peeled", "peeled more"))
def test_kd_replica_with_runs_at_the_cut(nbg, port, kind):
    xyz = [np.ascontiguousarray(v).astype(np.int32) for v in _cloud(kind)]
    tile = nbg.tile(*xyz)
    vind, nodes = nbg.kd_export(tile)
    tile.free()
    want = port.tree(*(U.syn.to_double(v) for v in xyz)).export()
    assert np.array_equal(vind.astype(np.uint64), want["vind"]), "point order"
    if kind.startswith("peeled"):  # past an eighth of the points, where the nodes' room is doubled
        assert (len(want["child1"]) > len(vind) // 8 + 1024) == (kind == "peeled more")
        return  # (more nodes than the export holds)
    inner, winner = nodes["child1"] >= 0, want["child1"] >= 0
    cuts = [sorted(zip(*(t[k][m].tolist() for k in ("divfeat", "divlow", "divhigh")))) for t, m in
            ((nodes, inner), (want, winner))]
    assert cuts[0] == cuts[1], "split planes"
    leaves = sorted(zip(nodes["begin"][~inner].tolist(), nodes["end"][~inner].tolist()))
    assert leaves == sorted(zip(want["left"][~winner].tolist(), want["right"][~winner].tolist())), "leaves"


def test_a_build_out_of_room_reads_no_node_it_did_not_write(nbg):
    """The nodes' room ends between the two nodes of a pair: the first has a
    place but is not written.  The context's cache is given blocks of the nodes'
    size that hold large numbers, which a reader would take for children."""
    xyz = [np.ascontiguousarray(v).astype(np.int32) for v in _cloud("peeled more")]
    stale = [nbg.tile(*[np.full(40_000, 2_000_000_000, np.int32)] * 3) for _ in range(4)]
    for tile in stale:
        tile.free()
    tile = nbg.tile(*xyz)
    vind, _ = nbg.kd_export(tile)
    assert np.array_equal(np.sort(vind), np.arange(len(vind)))
    tile.free()
