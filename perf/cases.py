"""Performance cases of the quadtree spatial join, through the package's public calls.

Eight families cover what a program does with the package:

  join       points and polygons on the device to rows, nothing kept between
             calls: quadtree_on_points -> polygon_bounding_boxes ->
             join_quadtree_and_bounding_boxes -> quadtree_point_in_polygon
  tree       the quadtree alone, as an application builds it once per layer
  pip        a kept quadtree joined with a new polygon layer
  nearest    a kept quadtree, nearest linestring of every point
  points     unindexed point_in_polygon, up to 31 polygons
  pairwise   point i against polygon i
  host       host columns to host rows in one call
  batched    many small joins planned together and run once

Sizes follow the package's own configurations (cuspatial_gb300/datasets.py)
and smaller and odd ones of the same shapes.  Inputs are drawn on the device
(host columns are copied back once) from torch generators seeded by the case's
seed; float cumulative sums are taken on integers, so that the same seed gives
the same bytes.

How many rows a join gives depends on its inputs.  The program these cases
stand for keeps the rows of a call in columns of its own, as long as its next
stage takes; the rest of those columns stays -1.
"""

import math

import numpy as np
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300.batched import BatchedPointInPolygon

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # a web request or a unit of a larger pipeline: latency and launches
        dict(name="join_1k_exact", family="join", points=1_003, polygons=17, vlo=4, vhi=40,
             extent=100.0, rlo=2.0, rhi=20.0, depth=5, max_size=32, clusters=0, dtype="float64",
             method="exact"),
        # the reference's CPU-runnable size (plain_small): default method
        dict(name="join_1m_exact", family="join", points=1_000_000, polygons=256, vlo=8, vhi=64,
             extent=1000.0, rlo=5.0, rhi=40.0, depth=7, max_size=128, clusters=0,
             dtype="float64", method="exact"),
        # float32 columns (sensor or rendering coordinates), clustered
        dict(name="join_3m_f32", family="join", points=3_000_017, polygons=2_001, vlo=8, vhi=128,
             extent=4000.0, rlo=2.0, rhi=60.0, depth=12, max_size=256, clusters=24,
             dtype="float32", method="exact"),
        # the index of a large point layer, with the points in its order
        dict(name="tree_50m", family="tree", points=50_000_000, extent=10000.0, depth=15,
             max_size=256, clusters=64, dtype="float64", ordered=True),
        # the precision configuration: the join step over a resident point layer
        dict(name="pip_100m_filtered", family="pip", points=100_000_000, polygons=100_000, vlo=8,
             vhi=512, extent=10000.0, rlo=2.0, rhi=60.0, depth=15, max_size=256, clusters=64,
             dtype="float64", method="filtered", ordered=True),
        # the same kind of join with the default method, as ported code calls it
        dict(name="pip_2m_exact", family="pip", points=2_000_003, polygons=10_000, vlo=8, vhi=256,
             extent=3162.0, rlo=2.0, rhi=60.0, depth=13, max_size=256, clusters=32,
             dtype="float64", method="exact", ordered=False),
        # snapping points to a road-like network: a crop of the package's own configuration
        dict(name="nearest_5m_filtered", family="nearest", points=5_000_000, linestrings=20_000,
             slo=2, shi=256, extent=3162.0, radius=25.0, depth=12, max_size=256,
             dtype="float64", method="filtered", ordered=True),
        # the same on a city block's worth of data, default method
        dict(name="nearest_20k_exact", family="nearest", points=20_011, linestrings=301,
             slo=2, shi=64, extent=300.0, radius=25.0, depth=8, max_size=64, dtype="float64",
             method="exact", ordered=False),
        # the reference benchmark's largest unindexed shape
        dict(name="points_10m_31", family="points", points=10_000_000, polygons=31, sides=100,
             dtype="float64", method="filtered"),
        # one point per polygon: a row-wise predicate over two columns
        dict(name="pairwise_1m", family="pairwise", points=1_000_000, vlo=4, vhi=400,
             dtype="float64", method="filtered"),
        # host table in, host table out
        dict(name="host_20m", family="host", points=20_000_000, polygons=20_000, vlo=8, vhi=256,
             extent=4472.0, rlo=2.0, rhi=60.0, depth=14, max_size=256, clusters=64,
             dtype="float64", method="filtered"),
        # one join per tile or customer, planned together, run once
        dict(name="batched_512", family="batched", instances=512, plo=1_000, phi=300_000, qlo=1,
             qhi=1_000, vlo=4, vhi=256, depth=5, max_size=256, method="filtered",
             ordered_index=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["join", "join", "tree", "pip", "pip", "nearest", "points", "pairwise",
                         "host", "batched"])
    dtype = rng.choice(["float64", "float64", "float64", "float32"])
    method = rng.choice(["exact", "filtered"])
    if family in ("join", "pip", "host"):
        hi = {"join": 20_000_000, "pip": 60_000_000, "host": 15_000_000}[family]
        n = _log(rng, 1_000, hi)
        q = _log(rng, 1, min(60_000, max(8, n // 50)))
        if method == "exact":  # the float64 method's cost grows with points x overlap
            n = min(n, 3_000_000)
        # up to about 3.6 polygons over a point, 2.3 in the listed cases
        extent = max(200.0, rng.uniform(25.0, 60.0) * math.sqrt(q))
        depth = max(3, min(15, int(math.log2(max(n, 64) / 64.0) / 2) + rng.randint(1, 6)))
        c = dict(family=family, points=n, polygons=q, vlo=rng.randint(4, 12),
                 vhi=rng.choice([32, 64, 200, 512]), extent=extent, rlo=2.0,
                 rhi=rng.uniform(10.0, 60.0), depth=depth, max_size=rng.choice([32, 100, 256, 512]),
                 clusters=rng.choice([0, 0, 16, 64]), dtype=dtype, method=method)
        if family == "pip":
            c["ordered"] = rng.random() < 0.5
        return c
    if family == "tree":
        return dict(family=family, points=_log(rng, 500, 50_000_000), extent=10000.0,
                    depth=rng.randint(4, 15), max_size=rng.choice([12, 64, 256, 1000]),
                    clusters=rng.choice([0, 8, 64]), dtype=dtype, ordered=rng.random() < 0.5)
    if family == "nearest":
        fast = method == "filtered" and dtype == "float64"  # others test every candidate
        lines = _log(rng, 40, 20_000 if fast else 400)
        n = _log(rng, 1_000, 4_000_000 if fast else 20_000)
        depth = max(3, min(14, int(math.log2(max(n, 64) / 64.0) / 2) + rng.randint(1, 4)))
        return dict(family=family, points=n, linestrings=lines, slo=2,
                    shi=rng.choice([16, 64, 256 if fast else 64]),
                    extent=max(50.0, 22.0 * math.sqrt(lines)), radius=rng.uniform(10.0, 25.0),
                    depth=depth, max_size=rng.choice([64, 256]), dtype=dtype, method=method,
                    ordered=rng.random() < 0.5)
    if family == "points":
        n = _log(rng, 1_000, 10_000_000 if method == "filtered" else 2_000_000)
        return dict(family=family, points=n, polygons=rng.randint(1, 31),
                    sides=_log(rng, 4, 1_000), dtype=dtype, method=method)
    if family == "pairwise":
        return dict(family=family, points=_log(rng, 500, 1_000_000), vlo=4,
                    vhi=rng.choice([8, 32, 128, 400]), dtype=dtype, method=method)
    return dict(family=family, instances=_log(rng, 8, 512), plo=_log(rng, 200, 1_000),
                phi=_log(rng, 20_000, 300_000), qlo=1, qhi=_log(rng, 10, 1_000), vlo=4,
                vhi=rng.choice([32, 256]), depth=rng.randint(4, 6),
                max_size=rng.choice([128, 256, 1024]), method="filtered",
                ordered_index=rng.random() < 0.25)


# -- inputs -----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(20261203 + 7919 * seed)


def _uni(g, n, lo, hi):
    return torch.rand(n, generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _ints(g, n, lo, hi):
    return torch.randint(lo, hi + 1, (n,), generator=g, device=DEV)


def _offsets(sizes):
    out = torch.zeros(sizes.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(sizes, 0, out=out[1:])
    return out


def _stars(g, cx, cy, k, radius, holes):
    """Star polygons of k vertices with per-vertex radius `radius(pid)`, rings
    closed; a share `holes` has the outer ring again, reversed and scaled by
    0.4.  Returns x, y, ring_offset, part_offset (device)."""
    p = cx.numel()
    pid = torch.repeat_interleave(torch.arange(p, device=DEV), k)
    vs = _offsets(k)
    # sorted uniform angles: exponential spacings on an integer grid
    e = (-torch.log1p(-torch.rand(pid.numel() + p, generator=g, device=DEV, dtype=F64)) *
         2.0 ** 20).long() + 1
    cum = torch.cumsum(e, 0)
    idx = torch.arange(pid.numel(), device=DEV) + pid  # one more spacing per polygon
    last = vs[1:] + torch.arange(p, device=DEV)
    base = cum[last] * 0
    base[1:] = cum[last[:-1]]
    ang = (cum[idx] - base[pid]).double() / (cum[last] - base)[pid].double()
    ang = (ang + _uni(g, p, 0.0, 1.0)[pid]) * (2.0 * math.pi)
    r = radius(pid)
    dx, dy = r * torch.cos(ang), r * torch.sin(ang)
    hole = torch.rand(p, generator=g, device=DEV, dtype=F64) < holes
    rings = 1 + hole.long()
    part = _offsets(rings)
    rp = torch.repeat_interleave(torch.arange(p, device=DEV), rings)
    inner = torch.arange(rp.numel(), device=DEV) != part[rp]
    ring = _offsets(k[rp] + 1)
    vr = torch.repeat_interleave(torch.arange(rp.numel(), device=DEV), k[rp] + 1)
    j = torch.arange(vr.numel(), device=DEV) - ring[vr]
    kk = k[rp][vr]
    j = torch.where(inner[vr], kk - j, j) % kk
    src = vs[rp[vr]] + j
    f = torch.where(inner[vr], 0.4, 1.0).to(F64)
    x = cx[rp[vr]] + f * dx[src]
    y = cy[rp[vr]] + f * dy[src]
    return x, y, ring.int(), part.int()


def _layer(g, c):
    q, ext = c["polygons"], c["extent"]
    cx, cy = _uni(g, q, 0.0, ext), _uni(g, q, 0.0, ext)
    k = _ints(g, q, c["vlo"], c["vhi"])
    rad = _uni(g, q, c["rlo"], c["rhi"])
    return _stars(g, cx, cy, k, lambda pid: rad[pid] * _uni(g, pid.numel(), 0.5, 1.0), 0.1)


def _points(g, c, layer=None):
    """Uniform or clustered points of [0, extent); with a layer, 1% of them on
    its vertices or within 1e-9 of an edge."""
    n, ext = c["points"], c["extent"]
    if c["clusters"]:
        m = c["clusters"]
        comp = _ints(g, n, 0, m - 1)
        sig = _uni(g, m, 0.001 * ext, 0.02 * ext)[comp]
        xy = []
        for _ in range(2):
            v = _uni(g, m, 0.0, ext)[comp]
            v += sig * torch.randn(n, generator=g, device=DEV, dtype=F64)
            xy.append(v.clamp_(0.0, math.nextafter(ext, 0.0)))
        x, y = xy
    else:
        x, y = _uni(g, n, 0.0, ext), _uni(g, n, 0.0, ext)
    nb = n // 100
    if layer is not None and nb:
        px, py, ring, _ = layer
        ring = ring.long()
        r = _ints(g, nb, 0, ring.numel() - 2)
        j = ring[r] + (_uni(g, nb, 0.0, 1.0) * (ring[r + 1] - ring[r] - 1)).long()
        t = _uni(g, nb, 0.0, 1.0)
        on_vertex = _uni(g, nb, 0.0, 1.0) < 0.5
        t[on_vertex] = 0.0
        ax, ay = px[j], py[j]
        ex, ey = px[j + 1] - ax, py[j + 1] - ay
        ln = torch.hypot(ex, ey).clamp_min_(1e-300)
        off = _uni(g, nb, -1e-9, 1e-9)
        off[on_vertex] = 0.0
        at = torch.arange(nb, device=DEV) * 100 + _ints(g, nb, 0, 99)
        hi = math.nextafter(ext, 0.0)
        x[at] = (ax + t * ex - ey / ln * off).clamp_(0.0, hi)
        y[at] = (ay + t * ey + ex / ln * off).clamp_(0.0, hi)
    return x, y


def _dtype(c):
    return torch.float32 if c["dtype"] == "float32" else F64


def _point_series(c, x, y):
    dt = _dtype(c)
    x, y = x.to(dt), y.to(dt)
    if "extent" in c and dt == torch.float32:  # rounding must not leave the box
        hi = c["extent"] * (1.0 - 2.0 ** -20)
        x, y = x.clamp_(max=hi), y.clamp_(max=hi)
    return cs.GeoSeries.from_points(x, y)


def _polygon_series(c, layer):
    x, y, ring, part = layer
    xy = torch.stack([x, y], 1).to(_dtype(c)).reshape(-1)
    return cs.GeoSeries.from_polygons_xy(xy, ring, part,
                                         torch.arange(part.numel(), dtype=torch.int32, device=DEV))


def _box(c):
    return 0.0, c["extent"], 0.0, c["extent"]


def _scale(c):
    return c["extent"] / (1 << c["depth"])


def _walks(g, c):
    """Random-walk linestrings: 2..shi segments of length U[1, 20], heading
    change N(0, 0.3).  Returns x, y, part_offset."""
    m, ext = c["linestrings"], c["extent"]
    k = _ints(g, m, c["slo"], c["shi"])
    lid = torch.repeat_interleave(torch.arange(m, device=DEV), k)
    seg = _offsets(k)

    def within(v):  # inclusive sums within each linestring, on a 2^-24 grid
        q = torch.cumsum(torch.round(v * 2.0 ** 24).long(), 0)
        base = torch.where(seg[:-1] > 0, q[seg[:-1] - 1], 0)
        return (q - base[lid]).double() * 2.0 ** -24

    step = _uni(g, lid.numel(), 1.0, 20.0)
    head = within(0.3 * torch.randn(lid.numel(), generator=g, device=DEV, dtype=F64))
    head += _uni(g, m, 0.0, 2.0 * math.pi)[lid]
    part = _offsets(k + 1)
    at = torch.arange(lid.numel(), device=DEV) + lid + 1
    out = []
    for d in (torch.cos(head), torch.sin(head)):
        s = _uni(g, m, 0.0, ext)
        v = torch.empty(int(part[-1]), dtype=F64, device=DEV)
        v[part[:-1]] = s
        v[at] = s[lid] + within(step * d)
        out.append(v)
    return out[0], out[1], part.int()


def _pairwise(g, c):
    n = c["points"]
    cx, cy = _uni(g, n, -1000.0, 1000.0), _uni(g, n, -1000.0, 1000.0)
    k = torch.exp(_uni(g, n, math.log(c["vlo"]), math.log(c["vhi"] + 1))).long()
    layer = _stars(g, cx, cy, k, lambda pid: _uni(g, pid.numel(), 1.0, 20.0), 0.1)
    ang, rad = _uni(g, n, 0.0, 2.0 * math.pi), _uni(g, n, 0.0, 25.0)
    x, y = cx + rad * torch.cos(ang), cy + rad * torch.sin(ang)
    # a tenth of the points on a vertex of their own polygon
    px, py, ring, part = layer
    b = torch.nonzero(_uni(g, n, 0.0, 1.0) < 0.1).reshape(-1)
    r0 = ring.long()[part.long()[b]]
    j = r0 + (_uni(g, b.numel(), 0.0, 1.0) * k[b]).long()
    x[b], y[b] = px[j], py[j]
    return x, y, layer


def _sizes(c):
    """Points and polygons of each instance: log-uniform, in no order and
    without relation to each other."""
    ni = c["instances"]

    def at(lo, hi, t):
        return max(lo, min(hi, int(lo * ((hi + 1) / lo) ** t)))

    return ([at(c["plo"], c["phi"], (i * 0.6180339887 + 0.31) % 1.0) for i in range(ni)],
            [at(c["qlo"], c["qhi"], (i * 0.4142135624 + 0.17) % 1.0) for i in range(ni)])


def _instances(g, c):
    ni = c["instances"]
    npts, npoly = (torch.tensor(v, device=DEV) for v in _sizes(c))
    side = _uni(g, ni, 100.0, 10000.0)
    ox, oy = _uni(g, ni, -50000.0, 50000.0), _uni(g, ni, -50000.0, 50000.0)
    po, qo = _offsets(npts), _offsets(npoly)
    pid = torch.repeat_interleave(torch.arange(ni, device=DEV), npts)
    below = 1.0 - 2.0 ** -40  # stays inside the instance's box after rounding
    x = ox[pid] + side[pid] * (_uni(g, pid.numel(), 0.0, 1.0) * below)
    y = oy[pid] + side[pid] * (_uni(g, pid.numel(), 0.0, 1.0) * below)
    qid = torch.repeat_interleave(torch.arange(ni, device=DEV), npoly)
    m = qid.numel()
    cx = ox[qid] + side[qid] * _uni(g, m, 0.05, 0.95)
    cy = oy[qid] + side[qid] * _uni(g, m, 0.05, 0.95)
    rad = side[qid] * _uni(g, m, 0.005, 0.05)
    layer = _stars(g, cx, cy, _ints(g, m, c["vlo"], c["vhi"]),
                   lambda v: rad[v] * _uni(g, v.numel(), 0.5, 1.0), 0.0)
    side, ox, oy = side.cpu().numpy(), ox.cpu().numpy(), oy.cpu().numpy()
    params = [(ox[i], ox[i] + side[i], oy[i], oy[i] + side[i], side[i] / (1 << c["depth"]),
               c["depth"], c["max_size"]) for i in range(ni)]
    po, qo = (t.cpu().numpy().astype(np.uint64) for t in (po, qo))
    return x, y, po, layer, qo, params


def prepare(case, seed):
    c, g = case, _gen(seed)
    s = {"case": c}
    f = c["family"]
    if f in ("join", "pip", "host"):
        layer = _layer(g, c)
        x, y = _points(g, c, layer)
        if f == "host":
            dt, pts = _dtype(c), _point_series(c, x, y).points
            px, py, ring, part = layer
            s["host"] = [t.cpu().pin_memory() for t in
                         (pts.x, pts.y, part, ring, px.to(dt), py.to(dt))]
            s["out"] = [torch.full((_capacity(c),), -1, dtype=torch.int32).pin_memory()
                        for _ in range(2)]
            return s
        s["points"], s["polygons"] = _point_series(c, x, y), _polygon_series(c, layer)
    elif f == "tree":
        s["points"] = _point_series(c, *_points(g, c))
        # an internal node holds more than max_size points, and has four children
        most = 4 * (c["points"] // (c["max_size"] + 1)) * c["depth"] + 4
        s["columns"] = _columns(most, torch.int32, torch.uint8, torch.bool, torch.int32,
                                torch.int32)
    elif f == "nearest":
        lx, ly, part = _walks(g, c)
        s["lines"] = cs.GeoSeries.from_linestrings_xy(
            torch.stack([lx, ly], 1).to(_dtype(c)).reshape(-1), part,
            torch.arange(part.numel(), dtype=torch.int32, device=DEV))
        s["points"] = _point_series(c, _uni(g, c["points"], 0.0, c["extent"]),
                                    _uni(g, c["points"], 0.0, c["extent"]))
    elif f == "points":
        n, q, m = c["points"], c["polygons"], c["sides"]
        x, y = _uni(g, n, -20.0, 20.0), _uni(g, n, -20.0, 20.0)
        a = (torch.arange(m + 1, device=DEV) % m).to(F64) * (2.0 * math.pi / m)
        xy = torch.stack([10.0 * torch.cos(a), 10.0 * torch.sin(a)], 1).to(_dtype(c))
        off = torch.arange(q + 1, dtype=torch.int32, device=DEV)
        s["points"] = cs.GeoSeries.from_points(x.to(_dtype(c)), y.to(_dtype(c)))
        s["polygons"] = cs.GeoSeries.from_polygons_xy(xy.repeat(q, 1).reshape(-1), off * (m + 1),
                                                      off, off)
    elif f == "pairwise":
        x, y, layer = _pairwise(g, c)
        s["points"] = cs.GeoSeries.from_points(x.to(_dtype(c)), y.to(_dtype(c)))
        s["polygons"] = _polygon_series(c, layer)
    else:
        x, y, po, layer, qo, params = _instances(g, c)
        px, py, ring, part = layer
        xy = torch.stack([px, py], 1).reshape(-1)
        polys = cs.GeoSeries.from_polygons_xy(
            xy, ring, part, torch.arange(part.numel(), dtype=torch.int32, device=DEV))
        s["batch"] = (x, y, po, polys, qo, params)
    if f in ("join", "pip", "batched"):
        s["columns"] = _columns(_capacity(c), torch.int32, torch.int32)
    if f in ("pip", "nearest"):
        args = (s["points"], *_box(c), _scale(c), c["depth"], c["max_size"])
        if c["ordered"]:
            s["index"], s["tree"], s["order"] = cs.quadtree_on_points_ordered(*args)
        else:
            s["index"], s["tree"] = cs.quadtree_on_points(*args)
            s["order"] = None
    return s


def _overlap(c):
    """Mean number of polygons over a point; a star of radius r covers about
    0.58 pi r^2."""
    r2 = (c["rlo"] ** 2 + c["rlo"] * c["rhi"] + c["rhi"] ** 2) / 3.0
    return c["polygons"] * 0.58 * math.pi * r2 / c["extent"] ** 2


def _capacity(c):
    """Rows the program's columns hold: half as many again as the mean, and
    one per point, for points that gather where polygons do."""
    if c["family"] == "batched":
        # radius 0.5% to 5% of the side, centres within the inner 90%
        return 4096 + int(sum(n * min(q, 2.0 * (0.58 * math.pi * 9.25e-4 / 0.81) * q + 1.0)
                              for n, q in zip(*_sizes(c))))
    return int(c["points"] * min(c["polygons"], 1.5 * _overlap(c) + 1.0)) + 4096


def _columns(n, *dtypes):
    return [torch.full((n,), 255 if d == torch.uint8 else 0 if d == torch.bool else -1, dtype=d,
                       device=DEV) for d in dtypes]


def _keep(columns, values):
    n = values[0].numel()
    for c, v in zip(columns, values):
        c[:n].copy_(v)
    return [n, columns]


def run(state):
    c = state["case"]
    f = c["family"]
    if f == "tree":
        build = cs.quadtree_on_points_ordered if c["ordered"] else cs.quadtree_on_points
        index, tree, *order = build(state["points"], *_box(c), _scale(c), c["depth"],
                                    c["max_size"])
        return [index, order, _keep(state["columns"], list(tree.values()))]
    if f in ("join", "pip"):
        pts, polys, order = state["points"], state["polygons"], state.get("order")
        if f == "join":
            index, tree = cs.quadtree_on_points(pts, *_box(c), _scale(c), c["depth"],
                                                c["max_size"])
        else:
            index, tree = state["index"], state["tree"]
        boxes = cs.polygon_bounding_boxes(polys)
        pairs = cs.join_quadtree_and_bounding_boxes(tree, boxes, *_box(c), _scale(c), c["depth"])
        rows = cs.quadtree_point_in_polygon(pairs, tree, index, pts, polys, method=c["method"],
                                            ordered_points=order)
        return [index, _keep(state["columns"], list(rows.values()))]
    if f == "nearest":
        boxes = cs.linestring_bounding_boxes(state["lines"], c["radius"])
        pairs = cs.join_quadtree_and_bounding_boxes(state["tree"], boxes, *_box(c), _scale(c),
                                                    c["depth"])
        return cs.quadtree_point_to_nearest_linestring(
            pairs, state["tree"], state["index"], state["points"], state["lines"],
            method=c["method"], ordered_points=state["order"])
    if f == "points":
        return cs.point_in_polygon_bitmask(state["points"], state["polygons"], c["method"])
    if f == "pairwise":
        return cs.pairwise_point_in_polygon(state["points"], state["polygons"], c["method"])
    if f == "host":
        a, b = state["out"]
        n = cs.point_in_polygon_join_host(*state["host"][:2], *_box(c), _scale(c), c["depth"],
                                          c["max_size"], *state["host"][2:], a, b,
                                          method=c["method"])
        return [n, a, b]
    with BatchedPointInPolygon(*state["batch"], method=c["method"],
                               ordered_index=c["ordered_index"]) as plan:
        offsets, polygon, point = plan.run().rows()
        return [offsets, _keep(state["columns"], [polygon, point])]


def _mean_vertices(c):
    return 0.5 * (c["vlo"] + c["vhi"]) + 1.0


def work(case):
    """Inputs read once and outputs written once.  The path has no contraction;
    its operations are the comparisons of each result bit, which are counted
    as one per output row (the rows of a join from the layer's mean overlap)."""
    c, f = case, case["family"]
    w = 8 if c.get("dtype", "float64") == "float64" else 4
    if f in ("join", "pip", "host"):
        n = c["points"]
        rows = n * _overlap(c)
        polys = c["polygons"] * (1.1 * _mean_vertices(c) * 2 * w + 8)
        kept = 4 * n if f == "join" else 0  # point_indices are an output of the whole join
        return dict(bytes=2 * w * n + polys + 8 * rows + kept, flops=max(1.0, rows))
    if f == "tree":
        n = c["points"]
        return dict(bytes=2 * w * n + 4 * n + (2 * w * n if c["ordered"] else 0), flops=2.0 * n)
    if f == "nearest":
        n = c["points"]
        lines = c["linestrings"] * (0.5 * (c["slo"] + c["shi"]) + 1.0) * 2 * w
        return dict(bytes=2 * w * n + lines + n * (8 + w), flops=10.0 * n)
    if f == "points":
        n = c["points"]
        return dict(bytes=2 * w * n + 4 * n + c["polygons"] * (c["sides"] + 1) * 2 * w,
                    flops=float(n * c["polygons"]))
    if f == "pairwise":
        n = c["points"]
        mean = (c["vhi"] + 1 - c["vlo"]) / math.log((c["vhi"] + 1) / c["vlo"]) + 1.0
        return dict(bytes=n * (2 * w + 1 + 1.1 * mean * 2 * w + 8), flops=1.1 * mean * n)
    pts, qs = _sizes(c)
    rows = sum(n * q * 0.58 * math.pi * 9.25e-4 for n, q in zip(pts, qs))
    return dict(bytes=16.0 * sum(pts) + sum(qs) * _mean_vertices(c) * 16 + 8 * rows,
                flops=max(1.0, rows))


# -- 64-bit values ------------------------------------------------------------

def exact(case, seed):
    """Distances of the nearest-linestring cases small enough for all point x
    segment distances; every other output is whole numbers."""
    c = case
    if c["family"] != "nearest":
        return None
    n = c["points"]
    segments = c["linestrings"] * 0.5 * (c["slo"] + c["shi"])
    if n * segments > 2e10:
        return None
    s = prepare(case, seed)
    ln = s["lines"].lines
    lx, ly, part = ln.x.double(), ln.y.double(), ln.part_offset.long()
    starts = torch.ones(lx.numel(), dtype=torch.bool, device=DEV)
    starts[part[1:] - 1] = False
    a = torch.nonzero(starts).reshape(-1)
    ax, ay = lx[a], ly[a]
    ex, ey = lx[a + 1] - ax, ly[a + 1] - ay
    ee = ex * ex + ey * ey
    index = s["index"].long()
    px, py = s["points"].points.x.double()[index], s["points"].points.y.double()[index]
    best = torch.empty(n, dtype=F64, device=DEV)
    chunk = max(1, int(1e8 // max(1, a.numel())))
    for i in range(0, n, chunk):
        dx = px[i:i + chunk, None] - ax
        dy = py[i:i + chunk, None] - ay
        t = ((dx * ex + dy * ey) / ee).clamp_(0.0, 1.0)
        dx -= t * ex
        dy -= t * ey
        best[i:i + chunk] = (dx * dx + dy * dy).min(1).values.sqrt_()
    if bool((best > c["radius"]).any()):  # a point may have no candidate: no value to give
        return None
    return {"distance": best, "point_index": None, "linestring_index": None}
