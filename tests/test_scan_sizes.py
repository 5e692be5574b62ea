"""The device-wide scan at the sizes where its launches change (one tile, the
blocks adding up the tiles before theirs, the scan of partials), through the
depth-1 quadtree, whose nodes are a compaction over all sorted points: node
keys, lengths and offsets against the oracle (exactly)."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import assert_tree_equal

pytestmark = pytest.mark.gpu

TILE, DIRECT = 2048, 4096


@pytest.mark.parametrize("n", [1, TILE - 1, TILE, TILE + 1, 300 * TILE + 5, DIRECT * TILE,
                               DIRECT * TILE + 1])
def test_depth_one_tree_at_scan_edges(n):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 8.0, (2, n)).astype(np.float32)
    args = (0.0, 8.0, 0.0, 8.0, 4.0, 1, 10)
    pi, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x, y), *args)
    assert_tree_equal(pi, tree, *O.quadtree_on_points(x, y, *args))
