"""point_in_polygon's bitmask call by its grid of cells and without: point counts
at the edges of a round, of a warp's rounds and of the grid's use, 1 to 31
polygons, boxes holding none to all of the points, points on vertices, edges and
level with them, far from the origin (cells no wider than the points' bounds),
zero, huge and not finite, a polygon beyond float32 and one not finite, against
the oracle (exactly)."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import gpu_polygons, to_np

pytestmark = pytest.mark.gpu


def _polygons(rng, count, at, unit, spread):
    from cuspatial_gb300.datasets import Polygons
    x, y, ro = [], [], [0]
    for i in range(count):
        c = at + rng.uniform(-spread, spread, 2) * unit
        if i % 3 == 1:  # vertical and horizontal edges
            w, h = rng.uniform(1, 9, 2) * unit
            vx, vy = c[0] + w * np.array([0, 1, 1, 0, 0.]), c[1] + h * np.array([0, 0, 1, 1, 0.])
        else:
            a = np.sort(rng.uniform(0, 2 * np.pi, int(rng.integers(3, 120))))
            d = rng.uniform(2, 9) * unit * rng.uniform(0.6, 1.0, len(a))
            vx, vy = c[0] + d * np.cos(a), c[1] + d * np.sin(a)
            vx, vy = np.append(vx, vx[0]), np.append(vy, vy[0])
        x.append(vx)
        y.append(vy)
        ro.append(ro[-1] + len(vx))
    i = np.arange(count + 1, dtype=np.int32)
    return Polygons(np.concatenate(x), np.concatenate(y), np.array(ro, np.int32), i, i)


@pytest.mark.parametrize("method", ["exact", "filtered"])
@pytest.mark.parametrize("n,count,at,unit,spread", [
    (1, 1, 0.0, 1.0, 1.0), (31, 2, 0.0, 1.0, 3.0), (33, 31, 5.0, 1.0, 8.0),
    (129, 7, 1.0e5, 1.0, 8.0), (4096, 31, 0.0, 1e-20, 2.0), (30_011, 16, -40.0, 1.0, 300.0),
    (65_535, 31, 0.0, 1.0, 8.0), (65_536, 31, 0.0, 1.0, 8.0), (131_072, 31, 0.0, 1.0, 8.0), (70_001, 1, 3.0, 1.0, 1.0),
    (131_073, 20, 2.0e8, 1.0, 8.0), (200_003, 31, -7.0, 1e-20, 12.0), (300_000, 9, 0.0, 1e30, 9.0),
    (900_001, 5, 0.0, 1.0, 8.0),
])
def test_bitmask(n, count, at, unit, spread, method):
    dtype = np.float64  # the grid serves float64 points
    rng = np.random.default_rng([n, count])
    P = _polygons(rng, count, at, unit, spread)
    if count == 20:
        P.x[P.ring_offset[4]] = np.nan
        P.y[P.ring_offset[9]] = 1e60
    P.x, P.y = P.x.astype(dtype), P.y.astype(dtype)
    x, y = (at + rng.uniform(-spread - 10, spread + 10, (2, n)) * unit).astype(dtype)
    j, kind = rng.integers(0, len(P.x), n), rng.random(n)
    x, y = np.where(kind < 0.1, P.x[j], x), np.where(kind < 0.2, P.y[j], y)
    j1, t = np.minimum(j + 1, len(P.x) - 1), rng.random(n).astype(dtype)
    on = (kind > 0.2) & (kind < 0.3)
    x = np.where(on, P.x[j] + t * (P.x[j1] - P.x[j]), x)
    y = np.where(on, P.y[j] + t * (P.y[j1] - P.y[j]), y)
    if n > 100:
        x[3::97], y[5::97], x[7::97] = np.nan, np.inf, -np.inf
        x[11::97], y[13::97] = 0.0, dtype(3e38)
    got = cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(x, y), gpu_polygons(P, dtype),
                                      method)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
