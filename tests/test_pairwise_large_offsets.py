"""Pairwise point in polygon where the float32 offsets are finite and their
products are not (from about 2^64 on; coordinates split into float32 parts up to
2^100): against the oracle."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from cuspatial_gb300.datasets import Polygons
from oracle import oracle as O

from helpers import gpu_polygons, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [1e17, 2.0 ** 60, 1e19, 2e19, 1e20, 1e21, 1e22, 1e28])
@pytest.mark.parametrize("lattice", [True, False])
def test_pairwise_products_beyond_float32(unit, lattice):
    rng = np.random.default_rng(7)
    n = 4000
    k = rng.integers(3, 9, n)
    ro = np.concatenate([[0], np.cumsum(k)]).astype(np.int32)

    def coordinates(m):
        return (rng.integers(-3, 4, m) if lattice else rng.uniform(-3, 3, m)) * unit

    px, py, x, y = (coordinates(m) for m in (ro[-1], ro[-1], n, n))
    ids = np.arange(n + 1, dtype=np.int32)
    P = Polygons(px, py, ro, ids, ids)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y, pairwise=True)
    for method in ("exact", "filtered"):
        got = to_np(cs.pairwise_point_in_polygon(cs.GeoSeries.from_points(x, y),
                                                 gpu_polygons(P), method))
        np.testing.assert_array_equal(got, want, err_msg=method)


def test_pairwise_example():
    # the first edge's cross product is -5e38, beyond float32
    P = Polygons(np.array([-3e19, 2e19, 3e19]), np.array([-2e19, 3e19, -3e19]),
                 np.array([0, 3], np.int32), np.array([0, 1], np.int32),
                 np.array([0, 1], np.int32))
    x, y = np.zeros(1), np.zeros(1)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y, pairwise=True)
    got = to_np(cs.pairwise_point_in_polygon(cs.GeoSeries.from_points(x, y), gpu_polygons(P),
                                             "filtered"))
    np.testing.assert_array_equal(got, want)
    assert want[0]
