"""The join at the sizes where its launches change: polygon counts around one
round and all rounds of the one-block index scans, and pair counts around the
one-block sort, against the oracle (exactly)."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from cuspatial_gb300.datasets import Polygons
from oracle import oracle as O

from helpers import gpu_polygons, to_np, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["exact", "filtered"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("count,n,max_size", [
    (1, 40, 4), (31, 900, 8), (1024, 1500, 64), (1025, 3000, 200), (1900, 2500, 2500),
    (4096, 2048, 300), (4097, 2049, 300),
])
def test_join_sizes(method, dtype, count, n, max_size):
    rng = np.random.default_rng([count, n])
    c, r = rng.uniform(0, 64, (count, 2)), rng.uniform(0.2, 1.5, (count, 1))
    k = 6
    a = np.sort(rng.uniform(0, 2 * np.pi, (count, k)), axis=1)
    px = np.concatenate([c[:, :1] + r * np.cos(a), c[:, :1] + r * np.cos(a[:, :1])], 1)
    py = np.concatenate([c[:, 1:] + r * np.sin(a), c[:, 1:] + r * np.sin(a[:, :1])], 1)
    ring = np.arange(0, (k + 1) * count + 1, k + 1, dtype=np.int32)
    part = np.arange(count + 1, dtype=np.int32)
    P = Polygons(px.reshape(-1).astype(dtype), py.reshape(-1).astype(dtype), ring, part, part)
    x, y = rng.uniform(0, 64, (2, n)).astype(dtype)
    args = (0.0, 64.0, 0.0, 64.0, 1.0, 6)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P, dtype)
    pi, tree = cs.quadtree_on_points(pts, *args, max_size)
    pairs = cs.join_quadtree_and_bounding_boxes(tree, cs.polygon_bounding_boxes(polys), *args)
    got = cs.quadtree_point_in_polygon(pairs, tree, pi, pts, polys, method=method)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    oj = O.join_quadtree_and_bounding_boxes(
        ot, O.polygon_bounding_boxes(part, ring, P.x, P.y), *args)
    for key in ("bbox_offset", "quad_offset"):
        np.testing.assert_array_equal(u32(pairs[key]), oj[key])
    want = O.quadtree_point_in_polygon(oj, ot, opi, x, y, part, ring, P.x, P.y)
    for key in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[key]), want[key].astype(np.int32))
