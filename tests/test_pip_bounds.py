"""The exact point-in-polygon join that compares float32 bounds before the
reference's float64 expression, against the oracle (exactly): points on vertices
and edges and within rounding of them, coordinates far from the origin (bounds
that decide little), at zero and beyond float32, vertical edges, points that are
not finite, one-slab and many-slab polygons, and device and host rows."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import gpu_polygons, to_np

pytestmark = pytest.mark.gpu

N = 70_000  # the bounds serve 65536 points on


def _polygons(rng, count, sizes, at, unit, boxes):
    from cuspatial_gb300.datasets import Polygons
    x, y, ro = [], [], [0]
    for i in range(count):
        c = at + rng.uniform(0, 20, 2) * unit
        k = int(rng.choice(sizes))
        if boxes and i % 2:  # axis-parallel: vertical and horizontal edges
            w, h = rng.uniform(0.5, 6, 2) * unit
            vx, vy = c[0] + w * np.array([0, 1, 1, 0, 0.]), c[1] + h * np.array([0, 0, 1, 1, 0.])
        else:
            a = np.sort(rng.uniform(0, 2 * np.pi, k))
            d = rng.uniform(0.3, 5.0) * unit * rng.uniform(0.5, 1.0, k)
            vx, vy = c[0] + d * np.cos(a), c[1] + d * np.sin(a)
            vx, vy = np.append(vx, vx[0]), np.append(vy, vy[0])
        x.append(vx)
        y.append(vy)
        ro.append(ro[-1] + len(vx))
    i = np.arange(count + 1, dtype=np.int32)
    return Polygons(np.concatenate(x), np.concatenate(y), np.array(ro, np.int32), i, i)


@pytest.mark.parametrize("at,unit,sizes,boxes,depth,max_size", [
    (0.0, 1.0, [3, 4, 7], True, 6, 32), (500.0, 1.0, [8, 60, 300], False, 7, 256),
    (-3.0e7, 1.0, [5, 40, 200], True, 5, 500), (0.0, 1e-30, [6, 90], True, 6, 64),
    (-7.0, 1.0, [1500], True, 3, 4000), (0.0, 1e37, [12, 50], True, 6, 100),
    (0.0, 1e60, [12, 50], True, 6, 100),
])
def test_exact_join_by_bounds(at, unit, sizes, boxes, depth, max_size):
    rng = np.random.default_rng([int(abs(at)), len(sizes), depth, max_size])
    P = _polygons(rng, 60, sizes, at, unit, boxes)
    x, y = at + rng.uniform(-3, 23, (2, N)) * unit
    j = rng.integers(0, len(P.x), N)
    kind = rng.random(N)
    on = kind < 0.1
    x, y = np.where(on, P.x[j], x), np.where(on, P.y[j], y)
    t, j1 = rng.random(N), np.minimum(j + 1, len(P.x) - 1)
    edge = (kind >= 0.1) & (kind < 0.2)  # on edges up to rounding
    x = np.where(edge, P.x[j] + t * (P.x[j1] - P.x[j]), x)
    y = np.where(edge, P.y[j] + t * (P.y[j1] - P.y[j]), y)
    level = (kind >= 0.2) & (kind < 0.3)  # level with a vertex, or at its x
    y = np.where(level & (t < 0.5), P.y[j], y)
    x = np.where(level & (t >= 0.5), P.x[j], x)
    lo, hi = at - 4 * unit, at + 24 * unit
    x[::9973], y[5::9973], x[7::9973], y[11::9973] = np.nan, np.inf, -np.inf, np.nan
    args = (lo, hi, lo, hi, (hi - lo) / (1 << depth), depth)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P)
    pi, tree = cs.quadtree_on_points(pts, *args, max_size)
    pairs = cs.join_quadtree_and_bounding_boxes(tree, cs.polygon_bounding_boxes(polys), *args)
    got = cs.quadtree_point_in_polygon(pairs, tree, pi, pts, polys)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    obb = O.polygon_bounding_boxes(P.part_offset, P.ring_offset, P.x, P.y)
    oj = O.join_quadtree_and_bounding_boxes(ot, obb, *args)
    want = O.quadtree_point_in_polygon(oj, ot, opi, x, y, P.part_offset, P.ring_offset, P.x, P.y)
    for k in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[k]), want[k].astype(np.int32))
    n = len(want["point_index"])
    out = [torch.full((n + 8,), -1, dtype=torch.int32).pin_memory() for _ in range(2)]
    cols = [torch.from_numpy(np.ascontiguousarray(v)) for v in
            (x, y, P.part_offset, P.ring_offset, P.x, P.y)]
    rows = cs.point_in_polygon_join_host(*cols[:2], *args, max_size, *cols[2:], *out)
    assert rows == n
    np.testing.assert_array_equal(out[0][:n].numpy(), want["polygon_index"].astype(np.int32))
    np.testing.assert_array_equal(out[1][:n].numpy(),
                                  opi[want["point_index"]].astype(np.int32))
