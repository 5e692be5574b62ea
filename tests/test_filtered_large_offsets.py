"""The float32 filter of the point-in-polygon join, of the bitmask call without
the grid of cells and of a batched plan, where offsets are finite in float32 and
their products are not (from about 2^64 on), against the oracle."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from cuspatial_gb300.batched import BatchedPointInPolygon
from oracle import oracle as O

from helpers import gpu_polygons, to_np
from test_pip_large_offsets import UNITS, join, join_oracle, layer, points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_size", [40, 600])
@pytest.mark.parametrize("unit", UNITS)
def test_filtered_join(unit, max_size):
    rng = np.random.default_rng(13)
    P = layer(rng, 40, unit)
    x, y = points(rng, P, 30_000, unit)
    a = (-4 * unit, 24 * unit, 6, max_size)
    got, want = join(x, y, P, *a, "filtered"), join_oracle(x, y, P, *a)
    for k in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[k]), want[k].astype(np.int32))


@pytest.mark.parametrize("unit", UNITS)
def test_filtered_bitmask(unit):
    rng = np.random.default_rng(14)
    P = layer(rng, 25, unit)
    x, y = points(rng, P, 30_000, unit)
    got = cs.point_in_polygon_bitmask(cs.GeoSeries.from_points(x, y), gpu_polygons(P),
                                      "filtered")
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("ordered_index", [False, True])
@pytest.mark.parametrize("unit", UNITS)
def test_filtered_batched_plan(unit, ordered_index):
    rng = np.random.default_rng(15)
    P = layer(rng, 40, unit)
    x, y = points(rng, P, 20_000, unit)
    lo, hi, depth, max_size = -4 * unit, 24 * unit, 5, 200
    import torch
    offs = np.array([0, len(x)], np.uint64), np.array([0, 40], np.uint64)
    with BatchedPointInPolygon(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), offs[0],
                               gpu_polygons(P), offs[1],
                               [(lo, hi, lo, hi, (hi - lo) / (1 << depth), depth, max_size)],
                               method="filtered", ordered_index=ordered_index) as plan:
        _, polygon, point = plan.run().rows()
        got = to_np(polygon), to_np(point)
    want = join_oracle(x, y, P, lo, hi, depth, max_size)
    for g, k in zip(got, ("polygon_index", "point_index")):
        np.testing.assert_array_equal(g, want[k].astype(np.int32))
