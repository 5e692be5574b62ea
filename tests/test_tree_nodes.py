"""Quadtree nodes of all levels from one pass over the sorted keys, against the
oracle (exactly): sizes at the edges of its position tiles, leaf sizes from one
point to more than the tree holds, repeated points (bottom leaves larger than
max_size), points outside the box, and every depth from the first the pass
serves."""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import assert_tree_equal

pytestmark = pytest.mark.gpu

E = 99.7  # cell sizes that are not representable


def _points(kind, n, rng, depth):
    if kind == "uniform":
        return rng.uniform(0, E, n), rng.uniform(0, E, n)
    if kind == "repeated":  # few distinct points, many of each
        k = rng.integers(0, max(1, n // 97) + 1, n)
        p = rng.uniform(0, E, (max(1, n // 97) + 1, 2))
        return p[k, 0], p[k, 1]
    if kind == "clustered":
        c = rng.uniform(0, E, (5, 2))[rng.integers(0, 5, n)]
        s = 10.0 ** rng.uniform(-6, 0, n)
        p = c + s[:, None] * rng.standard_normal((n, 2))
        return p[:, 0], p[:, 1]  # some lie outside the box
    if kind == "boundary":  # on cell boundaries, a few roundings to either side
        s = E / (1 << depth)
        p = rng.integers(0, (1 << depth) + 1, (2, n)) * s
        for _ in range(3):
            m = rng.random((2, n))
            p = np.where(m < 0.3, np.nextafter(p, -1.0), np.where(m < 0.6, np.nextafter(p, 2 * E), p))
        return np.clip(p, 0.0, E)
    x = rng.uniform(-0.2 * E, 1.2 * E, n)  # a ramp, partly outside
    return x, x + rng.uniform(0, 1e-3, n)


@pytest.mark.parametrize("kind", ["uniform", "repeated", "clustered", "ramp", "boundary"])
@pytest.mark.parametrize("n,depth,max_size", [
    (1, 2, 1), (2, 15, 1), (31, 5, 1), (255, 3, 2), (256, 15, 3), (2047, 15, 1), (2048, 4, 7),
    (2049, 15, 16), (4097, 7, 2047), (6143, 6, 2048), (6145, 12, 2049), (10_000, 2, 5),
    (10_000, 15, 20_000), (70_001, 13, 12), (300_007, 15, 256),
])
def test_tree_matches_oracle(kind, n, depth, max_size):
    rng = np.random.default_rng([n, depth, max_size, len(kind)])
    for dtype in (np.float64, np.float32):
        x, y = (v.astype(dtype) for v in _points(kind, n, rng, depth))
        scale = E / (1 << depth)
        args = (0.0, E, 0.0, E, scale, depth, max_size)
        pi, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x, y), *args)
        assert_tree_equal(pi, tree, *O.quadtree_on_points(x, y, *args))
