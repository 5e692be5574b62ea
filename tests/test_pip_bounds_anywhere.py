"""Float32 bounds of points and edges wherever the layer lies (projected and
geographic coordinates, small polygons over a large extent, a few polygons apart
from the others or without vertices): rows equal to the oracle's, and few
candidates left to float64."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from cuspatial_gb300.api import last_refined_count
from oracle import oracle as O

from helpers import gpu_polygons, to_np
from test_pip_large_offsets import join, join_oracle, layer, points

pytestmark = pytest.mark.gpu

PLACES = [(0.0, 1.0), (5.0e3, 1.0), (-4.5e6, 1.0), (48.2, 1e-5), (3.0e9, 1.0), (1e17, 1e5)]


@pytest.mark.parametrize("n,method", [(70_000, "exact"), (140_000, "filtered")])
@pytest.mark.parametrize("at,unit", PLACES)
def test_bitmask(at, unit, n, method):
    rng = np.random.default_rng(21)
    P = layer(rng, 25, unit, at)
    x, y = points(rng, P, n, unit, at)
    got = cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(x, y), gpu_polygons(P), method)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
    if method == "filtered" and at * 2.0 ** -44 < unit:
        # an eighth of the points are on or level with vertices; a point meets two
        # or three of the polygons' edges
        assert last_refined_count() < n // 2


@pytest.mark.parametrize("at,unit", PLACES)
def test_exact_join(at, unit):
    rng = np.random.default_rng(22)
    P = layer(rng, 40, unit, at)
    x, y = points(rng, P, 70_000, unit, at)
    a = (at - 4 * unit, at + 24 * unit, 6, 100)
    got, want = join(x, y, P, *a, "exact"), join_oracle(x, y, P, *a)
    for k in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[k]), want[k].astype(np.int32))


@pytest.mark.parametrize("outlier", [0.0, 1e12, 1e37, 1e60, -1e300])
@pytest.mark.parametrize("extent", [1e3, 1e7])
def test_small_polygons_over_a_large_extent(extent, outlier):
    # slabs far thinner than float32 resolves the extent: looked up in float64
    rng = np.random.default_rng(23)
    count, n = 31, 70_000
    P = layer(rng, count, 1.0)
    ids = np.repeat(np.arange(count), np.diff(P.ring_offset))
    move = rng.uniform(-extent, extent, (2, count))
    move[:, -1] += outlier
    P.x += move[0][ids]
    P.y += move[1][ids]
    j = rng.integers(0, count, n)
    k = P.ring_offset[j] + rng.integers(0, 10 ** 6, n) % np.diff(P.ring_offset)[j]
    spread = rng.choice([0.0, 1e-3, 3.0], n)
    x = P.x[k] + spread * rng.standard_normal(n)
    y = P.y[k] + spread * rng.standard_normal(n)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P)
    got = cs.point_in_polygon_bitmask(pts, polys, "exact")
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
    a = (-1.1 * extent, 1.1 * extent, 9, 50)
    got, want = join(x, y, P, *a, "exact"), join_oracle(x, y, P, *a)
    for c in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[c]), want[c].astype(np.int32))


@pytest.mark.parametrize("apart,n", [(0.0, 140_000), (60.0, 140_000), (60.0, 600_000),
                                     (1e5, 131_072), (1e5, 400_000), (1e300, 140_000)])
def test_filtered_bitmask_of_two_places(apart, n):
    # cells of the common box that tell the polygons apart, and ones that do not:
    # few candidates left to float64 either way
    rng = np.random.default_rng(24)
    P = layer(rng, 31, 1.0)
    second = np.repeat(np.arange(31) % 2 == 1, np.diff(P.ring_offset))
    P.x, P.y = P.x + apart * second, P.y + 0.3 * apart * second
    x, y = points(rng, P, n, 1.0)
    there = rng.random(n) < 0.5
    x, y = np.where(there, x + apart, x), np.where(there, y + 0.3 * apart, y)
    got = cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(x, y), gpu_polygons(P),
                                      "filtered")
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
    assert last_refined_count() < n or apart > 1e6


@pytest.mark.parametrize("sides", [2000, 30_000])
def test_filtered_bitmask_with_more_vertices_than_half_the_points(sides):
    rng = np.random.default_rng(sides)
    count, n = 5, 140_000
    a = np.linspace(0, 2 * np.pi, sides + 1)
    r = 8 * rng.uniform(0.9, 1.0, (count, sides))
    r = np.concatenate([r, r[:, :1]], 1)
    c = rng.uniform(-4, 4, (2, count, 1))
    x, y = (c[0] + r * np.cos(a)).ravel(), (c[1] + r * np.sin(a)).ravel()
    from cuspatial_gb300.datasets import Polygons
    i = np.arange(count + 1, dtype=np.int32)
    P = Polygons(x, y, (i * (sides + 1)).astype(np.int32), i, i)
    px, py = rng.uniform(-14, 14, (2, n))
    got, exact = (to_np(cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(px, py),
                                                    gpu_polygons(P), m)).view(np.uint32)
                  for m in ("filtered", "exact"))
    np.testing.assert_array_equal(got, exact)
    some = rng.integers(0, n, 3000)  # the oracle walks every edge
    want = O.point_in_polygon(px[some], py[some], P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(got[some], want.view(np.uint32))
