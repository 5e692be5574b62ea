"""The forest's nodes (one pass over tiles that never cross an instance) against
quadtree_on_points of each instance alone: instances of no point, one point and
sizes at the edges of a tile, depths 1 to 15 mixed, leaf sizes from one point to
more than the instance holds, repeated points; 32-bit and 64-bit sort keys."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300.batched import BatchedPointInPolygon

from helpers import assert_tree_equal, to_np, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depths", [(1, 2, 5), (15, 1, 9)])
def test_forest_matches_single_trees(depths):
    rng = np.random.default_rng(depths)
    sizes = [0, 1, 2047, 0, 2048, 2049, 5, 6145, 700, 0]
    po = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    x, y = rng.uniform(0, 10, (2, po[-1]))
    r = rng.integers(0, po[-1], po[-1] // 3)
    x[r], y[r] = x[r[0]], y[r[0]]  # many repeats of one point
    params = [(0.0, 10.0, 0.0, 10.0, 10.0 / (1 << depths[i % 3]), depths[i % 3],
               [1, 3, 64, 10_000][i % 4]) for i in range(len(sizes))]
    polys = cs.GeoSeries.from_polygons_xy(np.array([1., 1, 9, 1, 5, 9, 1, 1]), np.array([0, 4]),
                                          np.array([0, 1]), np.array([0, 1]))
    qo = np.zeros(len(sizes) + 1, np.uint64)
    qo[-1] = 1  # the polygon belongs to the last instance
    with BatchedPointInPolygon(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), po, polys,
                               qo, params) as plan:
        for i, p in enumerate(params):
            a, b = int(po[i]), int(po[i + 1])
            if a == b:
                assert plan.quadtree(i)["key"].numel() == 0
                continue
            pi, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x[a:b], y[a:b]), *p)
            t = {k: u32(tree[k]) for k in ("key", "length", "offset")}
            t["level"] = to_np(tree["level"])
            t["is_internal_node"] = to_np(tree["is_internal_node"]).astype(bool)
            assert_tree_equal(plan.point_indices(i), plan.quadtree(i), u32(pi), t)
