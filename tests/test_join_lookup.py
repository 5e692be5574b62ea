"""The box join's write pass (more pairs than are appended) where the nodes are
looked up by their first points, and where leaves share a first point, against the
oracle."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import u32

pytestmark = pytest.mark.gpu

E = 128.0


@pytest.mark.parametrize("count,n,depth,max_size,merge", [
    (400, 60_000, 12, 3, 0), (20_000, 3000, 5, 8, 0), (400, 60_000, 12, 3, 50),
    (400, 2_000_000, 15, 200, 0),
])
def test_write_pass(count, n, depth, max_size, merge):
    rng = np.random.default_rng([count, n, depth])
    x, y = rng.uniform(0, E, (2, n))
    args = (0.0, E, 0.0, E, E / (1 << depth), depth)
    _, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x, y), *args, max_size)
    _, ot = O.quadtree_on_points(x, y, *args, max_size)
    if merge:  # first points that several leaves share
        leaf = ~np.asarray(ot["is_internal_node"], bool)
        ot["offset"] = np.where(leaf, ot["offset"] // merge, ot["offset"]).astype(np.uint32)
        tree["offset"] = torch.from_numpy(ot["offset"].view(np.int32)).cuda().view(
            tree["offset"].dtype)
    lo = rng.uniform(-2, 2, (count, 2))
    b = np.concatenate([lo, lo + rng.uniform(E - 4, E + 4, (count, 2))], 1)
    cols = {k: np.ascontiguousarray(b[:, i]) for i, k in
            enumerate(("minx", "miny", "maxx", "maxy"))}
    got = cs.join_quadtree_and_bounding_boxes(
        tree, {k: torch.from_numpy(v).cuda() for k, v in cols.items()}, *args)
    want = O.join_quadtree_and_bounding_boxes(ot, cols, *args)
    box, node = u32(got["bbox_offset"]), u32(got["quad_offset"])
    assert len(box) > max(64 * count, 1 << 20)
    if merge:  # by first point, then as the boxes were walked
        key = ot["offset"][node]
        assert (np.diff(key.astype(np.int64)) >= 0).all()
        assert (np.diff(box.astype(np.int64))[np.diff(key.astype(np.int64)) == 0] >= 0).all()
        o, w = np.lexsort((node, box)), np.lexsort((want["quad_offset"], want["bbox_offset"]))
        box, node = box[o], node[o]
        want = {k: v[w] for k, v in want.items()}
    np.testing.assert_array_equal(box, want["bbox_offset"])
    np.testing.assert_array_equal(node, want["quad_offset"])
