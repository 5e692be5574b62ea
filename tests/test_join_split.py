"""The box join with several warps per box (few boxes over a large tree) against
the oracle (exactly): boxes over everything, over one leaf, over nothing and
across levels, trees of few and of many nodes at the level that is handed out,
and a tree whose node has more children than a stack holds (refused, as by one
warp)."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import u32

pytestmark = pytest.mark.gpu

E = 128.0


def _boxes(rng, count):
    lo = rng.uniform(-10, E, (count, 2))
    size = 10.0 ** rng.uniform(-3, 2.3, (count, 1))
    b = np.concatenate([lo, lo + size * rng.uniform(0.2, 1.0, (count, 2))], 1)
    b[0] = (-1, -1, E + 1, E + 1)
    if count > 2:
        b[1] = (E + 5, 0, E + 6, 1)
        b[2] = (E / 2, E / 2, E / 2, E / 2)
    return b


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("count,n,depth,max_size,clustered", [
    (1, 3000, 5, 4, False), (1, 200_000, 9, 8, False), (3, 200_000, 15, 8, True),
    (31, 60_000, 7, 1, False), (300, 60_000, 12, 16, True), (700, 20_000, 6, 2, False),
])
def test_few_boxes(dtype, count, n, depth, max_size, clustered):
    rng = np.random.default_rng([count, n, depth])
    p = rng.uniform(0, E, (n, 2))
    if clustered:
        p = np.clip(p[rng.integers(0, 3, n)] + rng.standard_normal((n, 2)) * 0.5, 0, E)
    x, y = p.T.astype(dtype)
    args = (0.0, E, 0.0, E, E / (1 << depth), depth)
    pi, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x, y), *args, max_size)
    b = _boxes(rng, count).astype(dtype)
    cols = {k: np.ascontiguousarray(b[:, i]) for i, k in
            enumerate(("minx", "miny", "maxx", "maxy"))}
    got = cs.join_quadtree_and_bounding_boxes(
        tree, {k: torch.from_numpy(v).cuda() for k, v in cols.items()}, *args)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    want = O.join_quadtree_and_bounding_boxes(ot, cols, *args)
    for k in ("bbox_offset", "quad_offset"):
        np.testing.assert_array_equal(u32(got[k]), want[k])


def test_too_many_children_are_refused():
    n = 3001
    i32 = lambda v: torch.from_numpy(np.asarray(v, np.int32)).cuda()  # noqa: E731
    tree = {"key": i32(np.concatenate([[0], np.arange(n - 1) % 4])),
            "level": torch.from_numpy(np.array([0] + [1] * (n - 1), np.uint8)).cuda(),
            "is_internal_node": torch.from_numpy(np.array([1] + [0] * (n - 1), bool)).cuda(),
            "length": i32([n - 1] + [1] * (n - 1)),
            "offset": i32(np.concatenate([[1], np.arange(n - 1)]))}
    box = {k: torch.tensor([v], dtype=torch.float64, device="cuda") for k, v in
           (("minx", 0.0), ("miny", 0.0), ("maxx", E), ("maxy", E))}
    with pytest.raises(RuntimeError):
        cs.join_quadtree_and_bounding_boxes(tree, box, 0.0, E, 0.0, E, E / 16, 4)
