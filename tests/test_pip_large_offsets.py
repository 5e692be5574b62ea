"""Point-in-polygon joins and the bitmask call where differences of coordinates
are finite in float32 and their products are not (from about 2^64 on), against
the oracle."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from cuspatial_gb300.datasets import Polygons
from oracle import oracle as O

from helpers import gpu_polygons, to_np

pytestmark = pytest.mark.gpu

UNITS = [1e16, 2.0 ** 58, 2e18, 1e19, 1e20, 1e21]


def layer(rng, count, unit, at=0.0):
    """Polygons of few, long edges (their lines pass the leaves at all distances)
    and of many vertices, in [0, 20] units."""
    x, y, ro = [], [], [0]
    for i in range(count):
        c = at + rng.uniform(4, 16, 2) * unit
        k = int(rng.integers(3, 6)) if i % 3 else 60
        a = np.sort(rng.uniform(0, 2 * np.pi, k))
        d = rng.uniform(1.0, 8.0) * unit * rng.uniform(0.4, 1.0, k)
        vx, vy = c[0] + d * np.cos(a), c[1] + d * np.sin(a)
        x.append(np.append(vx, vx[0]))
        y.append(np.append(vy, vy[0]))
        ro.append(ro[-1] + k + 1)
    i = np.arange(count + 1, dtype=np.int32)
    return Polygons(np.concatenate(x), np.concatenate(y), np.array(ro, np.int32), i, i)


def points(rng, P, n, unit, at=0.0):
    x, y = at + rng.uniform(-3, 23, (2, n)) * unit
    j, kind = rng.integers(0, len(P.x), n), rng.random(n)
    x, y = np.where(kind < 0.05, P.x[j], x), np.where(kind < 0.1, P.y[j], y)
    return x, y


def join(x, y, P, lo, hi, depth, max_size, method):
    args = (lo, hi, lo, hi, (hi - lo) / (1 << depth), depth)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P)
    pi, tree = cs.quadtree_on_points(pts, *args, max_size)
    pairs = cs.join_quadtree_and_bounding_boxes(tree, cs.polygon_bounding_boxes(polys), *args)
    return cs.quadtree_point_in_polygon(pairs, tree, pi, pts, polys, method=method)


def join_oracle(x, y, P, lo, hi, depth, max_size):
    args = (lo, hi, lo, hi, (hi - lo) / (1 << depth), depth)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    obb = O.polygon_bounding_boxes(P.part_offset, P.ring_offset, P.x, P.y)
    oj = O.join_quadtree_and_bounding_boxes(ot, obb, *args)
    return O.quadtree_point_in_polygon(oj, ot, opi, x, y, P.part_offset, P.ring_offset, P.x, P.y)


@pytest.mark.parametrize("unit", UNITS)
def test_exact_join(unit):
    rng = np.random.default_rng(11)
    P = layer(rng, 40, unit)
    x, y = points(rng, P, 70_000, unit)  # the bounds serve 65536 points on
    a = (-4 * unit, 24 * unit, 5, 300)
    got, want = join(x, y, P, *a, "exact"), join_oracle(x, y, P, *a)
    for k in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[k]), want[k].astype(np.int32))


@pytest.mark.parametrize("n,method", [(70_000, "exact"), (140_000, "filtered")])
@pytest.mark.parametrize("unit", UNITS)
def test_bitmask_by_cells(unit, n, method):
    rng = np.random.default_rng(12)
    P = layer(rng, 25, unit)
    x, y = points(rng, P, n, unit)
    got = cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(x, y), gpu_polygons(P), method)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
