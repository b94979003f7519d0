"""The workloads whose speed this repository is held to.

Each case is one pass of a user's program through the public entry points: a
fresh point set becomes a tile (Context.tile), its stages run (Context.run,
Context.run_columns or Context.run_batch) and the tile is freed, as a pipeline
does view after view with one long-lived Context.  The point sets are the
repository's synthetic airborne-lidar clouds (gpupdal_b200/synthetic.py: terrain,
buildings and vegetation; for the stress cloud exact duplicates and wires too),
drawn here on the GPU so that the large ones take milliseconds.  Coordinates are
LAS raw int32 at 0.01 m, in no spatial order.
"""
import functools
import math
import random

import numpy as np
import torch

from gpupdal_b200 import abi
from gpupdal_b200.native import Context, record_columns

SCALE = 0.01
RECORD = {"eigenvalues+normal": 64, "normal+covariancefeatures": 128}  # bytes per point


@functools.lru_cache(maxsize=None)
def _context():
    """The program's one context (device scratch and streams live in it)."""
    return Context(0)


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a thinned preview or a small crop: the call's fixed cost
        {"name": "normal_2k", "form": "device", "cloud": "terrain", "points": 2000,
         "density": 1.0, "stages": "normal", "knn": 8},
        # a small view handed over by a host pipeline stage: host arrays in and out
        {"name": "eigen_host_20k", "form": "host", "cloud": "mixture", "points": 20011,
         "density": 16.0, "stages": "eigenvalues", "knn": 32},
        # filters.normal knn=8 on the 250k-point terrain of the first benchmark configuration
        {"name": "normal_250k", "form": "device", "cloud": "terrain", "points": 250000,
         "density": 1.0, "stages": "normal", "knn": 8},
        # local outlier factor: the ordered neighbour lists
        {"name": "lof_500k", "form": "device", "cloud": "mixture", "points": 500009,
         "density": 16.0, "stages": "lof", "knn": 10},
        # features over each point's own optimal neighbourhood
        {"name": "optimized_700k", "form": "device", "cloud": "mixture", "points": 700001,
         "density": 16.0, "stages": "optimized", "knn": 14},
        # a mid-sized odd tile with duplicates and wires, two stages in one pass
        {"name": "stress_1m", "form": "records", "cloud": "stress", "points": 1000003,
         "density": 128.0, "stages": "eigenvalues+normal", "knn": 16},
        # a radius neighbourhood
        {"name": "radius_1m", "form": "device", "cloud": "mixture", "points": 1048573,
         "density": 16.0, "stages": "radius", "knn": 8},
        # the largest neighbour count of the served mix
        {"name": "eigen_knn64_1m5", "form": "device", "cloud": "mixture", "points": 1500001,
         "density": 16.0, "stages": "eigenvalues", "knn": 64},
        # filters.covariancefeatures knn=10 feature_set=all on 4M points (second configuration)
        {"name": "features_4m", "form": "device", "cloud": "mixture", "points": 4000000,
         "density": 16.0, "stages": "covariancefeatures", "knn": 10},
        # pinned host records in and out, end to end
        {"name": "stress_host_6m", "form": "pinned", "cloud": "stress", "points": 6000001,
         "density": 128.0, "stages": "eigenvalues+normal", "knn": 16},
        # many tiles of uneven size and knn in one call (a tenth of the batched configuration)
        {"name": "batch_24", "form": "batch", "cloud": "mixture", "points": 200000,
         "density": 16.0, "stages": "normal+covariancefeatures", "knn": 0, "tiles": 24},
        # eigenvalues + normal knn=16 on the 32M-point stress tile (third configuration)
        {"name": "stress_32m", "form": "records", "cloud": "stress", "points": 32000000,
         "density": 128.0, "stages": "eigenvalues+normal", "knn": 16},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes spread over their logarithm, any neighbour count."""
    kind = rng.choice(("one", "one", "one", "two", "two", "host", "other", "batch"))
    cloud = rng.choice(("terrain", "mixture", "mixture", "stress"))
    density = {"terrain": 1.0, "mixture": 16.0, "stress": 128.0}[cloud] * math.exp(rng.uniform(-0.7, 0.7))
    knn = rng.choice((rng.randint(3, 12), rng.randint(8, 20), rng.randint(16, 64)))
    density = round(density, 3)
    if kind == "one":
        return {"form": "device", "cloud": cloud, "points": _log_size(rng, 1500, 1.2e8 / (knn + 8)),
                "density": density, "knn": knn,
                "stages": rng.choice(("normal", "eigenvalues", "covariancefeatures"))}
    if kind == "two":
        return {"form": "records", "cloud": cloud, "points": _log_size(rng, 1500, 2e8 / (knn + 8)),
                "density": density, "knn": knn,
                "stages": rng.choice(("eigenvalues+normal", "normal+covariancefeatures"))}
    if kind == "host":
        form = rng.choice(("host", "pinned"))
        return {"form": form, "cloud": cloud, "density": density, "knn": knn,
                "points": _log_size(rng, 1500, 1000000 if form == "host" else 6000000),
                "stages": "eigenvalues" if form == "host" else "eigenvalues+normal"}
    if kind == "other":
        return {"form": "device", "cloud": "mixture", "points": _log_size(rng, 1500, 2000000),
                "density": 16.0, "knn": rng.randint(6, 14),
                "stages": rng.choice(("lof", "optimized", "radius"))}
    return {"form": "batch", "cloud": "mixture", "points": _log_size(rng, 15000, 200000),
            "density": 16.0, "stages": "normal+covariancefeatures", "knn": 0,
            "tiles": rng.randint(3, 30)}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _terrain_z(x, y):
    return 20.0 * torch.sin(x / 80.0) * torch.cos(y / 60.0)


def _mixture(gen, n, side):
    """60 % terrain, 25 % faces of boxes, 15 % vegetation blobs, metres."""
    def uni(m, lo, hi):
        return torch.rand(m, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    def nrm(m, s):
        return torch.randn(m, generator=gen, device="cuda", dtype=torch.float64) * s

    nt, nb = int(round(0.60 * n)), int(round(0.25 * n))
    nv = n - nt - nb
    x, y = uni(nt, 0.0, side), uni(nt, 0.0, side)
    parts = [torch.stack((x, y, _terrain_z(x, y) + nrm(nt, 0.05)))]
    boxes = max(1, int(round(400 * (side / 500.0) ** 2)))
    cx, cy = uni(boxes, 0.0, side), uni(boxes, 0.0, side)
    wx, wy, h = uni(boxes, 10.0, 40.0), uni(boxes, 10.0, 40.0), uni(boxes, 5.0, 30.0)
    z0 = _terrain_z(cx, cy)
    area = torch.stack((wx * wy, wy * h, wy * h, wx * h, wx * h), 1).reshape(-1)
    cum = torch.cumsum(area, 0)
    f = torch.searchsorted(cum, uni(nb, 0.0, 1.0) * cum[-1]).clamp_(max=5 * boxes - 1)
    b, f = f // 5, f % 5
    u, v = uni(nb, 0.0, 1.0), uni(nb, 0.0, 1.0)
    px = torch.where(f == 1, torch.zeros_like(u), torch.where(f == 2, torch.ones_like(u), u))
    py = torch.where(f == 3, torch.zeros_like(u), torch.where(f == 4, torch.ones_like(u),
                                                               torch.where(f == 0, v, u)))
    pz = torch.where(f == 0, torch.ones_like(v), v)
    parts.append(torch.stack((cx[b] - wx[b] / 2 + px * wx[b] + nrm(nb, 0.02),
                              cy[b] - wy[b] / 2 + py * wy[b] + nrm(nb, 0.02),
                              z0[b] + pz * h[b] + nrm(nb, 0.02))))
    blobs = max(8, int(2000 * (side / 500.0) ** 2))
    bx, by = uni(blobs, 0.0, side), uni(blobs, 0.0, side)
    bz, bs = _terrain_z(bx, by) + uni(blobs, 5.0, 20.0), uni(blobs, 1.0, 4.0)
    b = torch.randint(0, blobs, (nv,), generator=gen, device="cuda")
    parts.append(torch.stack((bx[b] + nrm(nv, 1.0) * bs[b], by[b] + nrm(nv, 1.0) * bs[b],
                              bz[b] + nrm(nv, 1.0) * bs[b])))
    return torch.cat(parts, 1)


def _cloud(cloud, n, density, seed):
    """x, y, z raw int32 CUDA tensors of n points."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    side = math.sqrt(n / density)

    def uni(m, lo, hi):
        return torch.rand(m, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    if cloud == "terrain":
        x, y = uni(n, 0.0, side), uni(n, 0.0, side)
        z = _terrain_z(x, y) + torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) * 0.05
        p = torch.stack((x, y, z))
    elif cloud == "mixture":
        p = _mixture(gen, n, side)
    else:
        # 2 % exact duplicates, 3 % points on wires
        nd, nw = int(round(0.02 * n)), int(round(0.03 * n))
        base = _mixture(gen, n - nd - nw, side)
        wires = max(4, int(round(400 * (side / 500.0) ** 2)))
        a = torch.stack((uni(wires, 0.0, side), uni(wires, 0.0, side), uni(wires, 10.0, 25.0)))
        b = torch.stack((uni(wires, 0.0, side), uni(wires, 0.0, side), uni(wires, 10.0, 25.0)))
        w = torch.randint(0, wires, (nw,), generator=gen, device="cuda")
        wp = a[:, w] + (b[:, w] - a[:, w]) * uni(nw, 0.0, 1.0)
        src = torch.randint(0, base.shape[1], (nd,), generator=gen, device="cuda")
        p = torch.cat((base, wp, base[:, src]), 1)
    p = p[:, torch.randperm(n, generator=gen, device="cuda")]
    p = torch.round(p / SCALE).to(torch.int32)
    return p[0].contiguous(), p[1].contiguous(), p[2].contiguous()


def _optimal(n, lo, hi, seed):
    """OptimalKNN (whole numbers in [lo, hi]) and OptimalRadius columns."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 7919)
    k = torch.randint(lo, hi + 1, (n,), generator=gen, device="cuda").to(torch.float64)
    r = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * 1.2 + 0.3
    return k, r


def _stages(kind, knn):
    if kind == "normal":
        return [abi.make_opts(abi.STAGE_NORMAL, knn=knn)]
    if kind == "eigenvalues":
        return [abi.make_opts(abi.STAGE_EIGENVALUES, knn=knn)]
    if kind == "covariancefeatures":
        return [abi.make_opts(abi.STAGE_COVARIANCEFEATURES, knn=knn, feature_mask=abi.FEAT_ALL)]
    if kind == "eigenvalues+normal":
        return _stages("eigenvalues", knn) + _stages("normal", knn)
    if kind == "normal+covariancefeatures":
        return _stages("normal", knn) + _stages("covariancefeatures", knn)
    if kind == "optimized":
        return [abi.make_opts(abi.STAGE_COVARIANCEFEATURES, knn=knn, feature_mask=abi.FEAT_ALL,
                              optimized=True)]
    if kind == "radius":
        return [abi.make_opts(abi.STAGE_NORMAL, knn=knn, radius=0.5)]
    return [abi.consumer_opts(abi.STAGE_LOF, minpts=knn)]


def _batch_tiles(case):
    """(points, knn) of a batch's tiles: log-normal sizes, knn of {8, 16, 32}."""
    rng = random.Random(case["tiles"] * 1000003 + case["points"])
    hi = min(4000000, 20 * case["points"])
    return [(int(min(hi, max(20000, math.exp(rng.gauss(math.log(case["points"]), 1.0))))),
             rng.choice((8, 16, 32))) for _ in range(case["tiles"])]


def _records(n, stages, size, device):
    """One zeroed record of `size` bytes per point and its column descriptions."""
    if device:
        rec = torch.zeros((n, size // 8), dtype=torch.float64, device="cuda")
    else:
        rec = torch.zeros((n, size // 8), dtype=torch.float64).pin_memory()
    return rec, record_columns(rec.data_ptr(), stages, size, 1 if device else 2)


def prepare(case, seed):
    ctx = _context()
    form, n = case["form"], case["points"]
    if form == "batch":
        tiles = []
        for i, (m, knn) in enumerate(_batch_tiles(case)):
            st = _stages(case["stages"], knn)
            rec, cols = _records(m, st, RECORD[case["stages"]], True)
            tiles.append({"xyz": _cloud(case["cloud"], m, case["density"], seed * 1000 + i),
                          "stages": st, "rec": rec, "cols": cols,
                          "optimal": _optimal(m, knn, knn, seed * 1000 + i)})
        return {"form": form, "ctx": ctx, "tiles": tiles}
    st = _stages(case["stages"], case["knn"])
    xyz = _cloud(case["cloud"], n, case["density"], seed)
    s = {"form": form, "ctx": ctx, "stages": st, "xyz": xyz, "optimal": (None, None)}
    if case["stages"] in ("covariancefeatures", "normal+covariancefeatures"):
        s["optimal"] = _optimal(n, case["knn"], case["knn"], seed)
    if case["stages"] == "optimized":
        s["optimal"] = _optimal(n, max(4, case["knn"] - 4), case["knn"], seed)
    if form == "records":
        s["rec"], s["cols"] = _records(n, st, RECORD[case["stages"]], True)
    elif form == "pinned":
        # packed records, as a PDAL row holds them; coordinates page-locked too
        s["rec"], s["cols"] = _records(n, st, 8 * sum(len(abi.stage_dims(o)) for o in st), False)
        s["pins"] = [v.cpu().pin_memory() for v in xyz]
        s["xyz"] = [v.numpy() for v in s["pins"]]
    elif form == "host":
        s["xyz"] = [v.cpu().numpy() for v in xyz]
        s["out"] = [np.zeros((len(abi.stage_dims(o)), n)) for o in st]
    else:
        s["out"] = [torch.zeros((len(abi.stage_dims(o)), n), dtype=torch.float64, device="cuda")
                    for o in st]
    return s


def run(state):
    ctx = state["ctx"]
    if state["form"] == "batch":
        ts = state["tiles"]
        tiles = [ctx.tile(*t["xyz"]) for t in ts]
        exc, _ = ctx.run_batch(tiles, [t["stages"] for t in ts], [t["cols"] for t in ts],
                               [t["optimal"] for t in ts])
        for tile in tiles:
            tile.free()
        return {"records": [t["rec"] for t in ts], "exceptions": sum(len(e) for e in exc)}
    tile = ctx.tile(*state["xyz"])
    kopt, ropt = state["optimal"]
    if state["form"] in ("records", "pinned"):
        exc, _ = ctx.run_columns(tile, state["stages"], state["cols"], optimal_knn=kopt,
                                 optimal_radius=ropt, aux_on_device=kopt is not None)
        tile.free()
        return {"records": state["rec"], "exceptions": len(exc)}
    outs, exc, _ = ctx.run(tile, state["stages"], optimal_knn=kopt, optimal_radius=ropt,
                           device_out=state["form"] == "device", out=state["out"])
    tile.free()
    return {"columns": outs, "exceptions": len(exc)}


# --------------------------------------------------------------------------
# what a pass cannot do without, and its values in 64 bits
# --------------------------------------------------------------------------
def _dims(kind):
    return sum(len(abi.stage_dims(o)) for o in _stages(kind, 8))


def work(case):
    """Coordinates read once, outputs (and optimal columns) moved once; the
    distances and second moments of the K neighbours and one 3x3 eigensolve."""
    tiles = _batch_tiles(case) if case["form"] == "batch" else [(case["points"], case["knn"])]
    aux = 16 if "covariancefeatures" in case["stages"] or case["stages"] == "optimized" else 0
    nbytes = sum(n * (12 + aux + 8 * _dims(case["stages"])) for n, _ in tiles)
    flops = sum(n * ((k + 1) * 26 + 250) for n, k in tiles)
    return {"bytes": nbytes, "flops": flops}


def _nearest(xyz, k):
    """Ids of the k nearest by FP64 distance of the scaled coordinates."""
    p = torch.stack(xyz, 1).to(torch.float64) * SCALE
    n = p.shape[0]
    step = max(1, (1 << 27) // n)
    out = []
    for r in range(0, n, step):
        q = p[r:r + step]
        d = (q[:, None, 0] - p[None, :, 0]) ** 2
        d += (q[:, None, 1] - p[None, :, 1]) ** 2
        d += (q[:, None, 2] - p[None, :, 2]) ** 2
        out.append(torch.topk(d, k, dim=1, largest=False, sorted=False).indices)
    return torch.cat(out)


def _eigen(xyz, k):
    """Eigenvalues (n, 3) ascending and vectors (n, 3, 3) of the covariances."""
    p = torch.stack(xyz, 1).to(torch.float64)
    c = []
    for ids in _nearest(xyz, k).split(1 << 20):
        d = p[ids]
        d = d - d.mean(1, keepdim=True)
        c.append(torch.einsum("rki,rkj->rij", d, d) * (SCALE * SCALE / (k - 1)))
    return np.linalg.eigh(torch.cat(c).cpu().numpy())


def _stage_exact(kind, w, v, optimal):
    if kind == "eigenvalues":
        return np.ascontiguousarray(w.T)
    if kind == "normal":
        nv = np.where(v[:, 2:3, 0] < 0, -1.0, 1.0) * v[:, :, 0]
        s = w.sum(1)
        return np.concatenate((nv.T, np.abs(w[:, 0] / s)[None]))
    l0, l1, l2 = (np.maximum(w[:, i], 0.0) for i in (2, 1, 0))
    s = l0 + l1 + l2
    l0, l1, l2 = np.sqrt(l0), np.sqrt(l1), np.sqrt(l2)
    a = np.abs(v)
    u = l0[:, None] * a[:, :, 2] + l1[:, None] * a[:, :, 1] + l2[:, None] * a[:, :, 0]
    k, r = (t.cpu().numpy() for t in optimal)
    with np.errstate(all="ignore"):
        return np.stack((
            (l0 - l1) / l0, (l1 - l2) / l0, l2 / l0, u[:, 2] / np.sqrt((u * u).sum(1)),
            np.cbrt(l2 * l1 * l0), (l0 - l2) / l0,
            -(l2 * np.log(l2) + l1 * np.log(l1) + l0 * np.log(l0)), s, l2 / s,
            1.0 - a[:, 2, 0], (k + 1.0) / (4.0 / 3.0 * 3.14159265 * r ** 3)))


def exact(case, seed):
    n, kind = case["points"], case["stages"]
    if case["form"] == "batch" or n > 300000 or kind in ("lof", "optimized", "radius"):
        return None
    xyz = _cloud(case["cloud"], n, case["density"], seed)
    w, v = _eigen(xyz, case["knn"] + 1)
    opt = _optimal(n, case["knn"], case["knn"], seed) if "covariancefeatures" in kind else None
    cols = [_stage_exact(one, w, v, opt) for one in kind.split("+")]
    if case["form"] in ("records", "pinned"):
        size = RECORD[kind] // 8 if case["form"] == "records" else sum(len(c) for c in cols)
        rec = np.zeros((n, size))
        rec[:, :sum(len(c) for c in cols)] = np.concatenate(cols).T
        return {"records": rec, "exceptions": None}
    return {"columns": cols, "exceptions": None}
