"""Nearest linestrings with candidates passed over by their bounding boxes,
against the oracle bit for bit: linestrings of one point to several chunks of 8
segments, points on vertices and on axis-parallel segments (zero distances,
which the reference's fold passes over), repeated linestrings (ties by id),
coordinates far from the origin, and more points per leaf than one round of a
warp.  A linestring or a point that is not finite prunes nothing.  (The float32
filter's own zero-distance rules have their adversarial test; where a point lies
within rounding of a segment's inside and the reference's square comes out
negative, its fold starts again, which the filter does not follow.)"""

import numpy as np
import pytest

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import to_np, u32

pytestmark = pytest.mark.gpu


def _lines(rng, sizes, at, ext):
    x, y, part = [], [], [0]
    for i, k in enumerate(sizes):
        if i % 7 == 3 and i > 3:  # the same linestring again
            vx, vy = x[-1], y[-1]
        else:
            p = at + rng.uniform(0, ext, 2)
            step = rng.uniform(-1, 1, (k, 2)) * (1.0 if i % 5 else 0.0 if k < 3 else 8.0)
            step[::3, 0] = 0.0  # axis-parallel pieces
            v = p + np.cumsum(step, 0)
            vx, vy = v[:, 0], v[:, 1]
        x.append(vx)
        y.append(vy)
        part.append(part[-1] + len(vx))
    return np.concatenate(x), np.concatenate(y), np.array(part, np.int32)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,sizes,at,max_size", [
    (1, [2], 0.0, 8), (40, [1, 2, 9, 10], 0.0, 64), (700, [2, 8, 9, 17, 33] * 5, 0.0, 16),
    (3000, [2, 3, 70, 300] * 12, 4096.0, 500), (3000, [2, 40] * 30, -1.0e6, 64),
])
def test_nearest_with_pruning(dtype, n, sizes, at, max_size):
    rng = np.random.default_rng([n, len(sizes), max_size])
    ext = 40.0
    lx, ly, part = _lines(rng, sizes, at, ext)
    lx, ly = lx.astype(dtype), ly.astype(dtype)
    x, y = (at + rng.uniform(0, ext, (2, n))).astype(dtype)
    j = rng.integers(0, len(lx), n)
    on = rng.random(n) < 0.3
    x, y = np.where(on, lx[j], x), np.where(on, ly[j], y)
    mid = (rng.random(n) < 0.1) & (j + 1 < len(lx))  # on a vertical segment's inside
    y = np.where(mid, ((ly[j] + ly[np.minimum(j + 1, len(ly) - 1)]) / 2).astype(dtype), y)
    x = np.where(mid, lx[j], x)
    lo, hi = at - 2 * ext, at + 3 * ext
    args = (lo, hi, lo, hi, (hi - lo) / 64, 6)
    pts = cs.GeoSeries.from_points(x, y)
    xy = np.empty(2 * len(lx), dtype)
    xy[0::2], xy[1::2] = lx, ly
    ls = cs.GeoSeries.from_linestrings_xy(xy, part, np.arange(len(part), dtype=np.int32))
    pi, tree = cs.quadtree_on_points(pts, *args, max_size)
    bb = cs.linestring_bounding_boxes(ls, 3 * ext)
    pairs = cs.join_quadtree_and_bounding_boxes(tree, bb, *args)
    got = cs.quadtree_point_to_nearest_linestring(pairs, tree, pi, pts, ls)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    obb = O.linestring_bounding_boxes(part, lx, ly, 3 * ext)
    oj = O.join_quadtree_and_bounding_boxes(ot, obb, *args)
    want = O.quadtree_point_to_nearest_linestring(oj, ot, opi, x, y, part, lx, ly)
    np.testing.assert_array_equal(u32(got["point_index"]), want["point_index"])
    np.testing.assert_array_equal(u32(got["linestring_index"]), want["linestring_index"])
    np.testing.assert_array_equal(to_np(got["distance"]), want["distance"])


@pytest.mark.parametrize("method", ["exact", "filtered"])
def test_nearest_prunes_nothing_without_finite_bounds(method):
    rng = np.random.default_rng(5)
    n, part = 400, np.arange(0, 21 * 12, 12, dtype=np.int32)
    lx, ly = rng.uniform(0, 40, (2, part[-1]))
    lx[17], ly[40] = np.nan, np.inf
    x, y = rng.uniform(0, 40, (2, n))
    args = (0.0, 40.0, 0.0, 40.0, 40 / 16, 4)
    pts = cs.GeoSeries.from_points(x, y)
    xy = np.stack([lx, ly], 1).reshape(-1)
    ls = cs.GeoSeries.from_linestrings_xy(xy, part, np.arange(len(part), dtype=np.int32))
    pi, tree = cs.quadtree_on_points(pts, *args, 32)
    opi, ot = O.quadtree_on_points(x, y, *args, 32)
    q = np.flatnonzero(~ot["is_internal_node"])
    nl = len(part) - 1
    pairs = {"bbox_offset": np.tile(np.arange(nl, dtype=np.int32), len(q)),
             "quad_offset": np.repeat(q.astype(np.int32), nl)}
    order = np.argsort(ot["offset"][pairs["quad_offset"]], kind="stable")
    pairs = {k: v[order] for k, v in pairs.items()}
    import torch
    gp = {k: torch.from_numpy(v).cuda() for k, v in pairs.items()}
    got = cs.quadtree_point_to_nearest_linestring(gp, tree, pi, pts, ls, method=method)
    want = O.quadtree_point_to_nearest_linestring(pairs, ot, opi, x, y, part, lx, ly)
    np.testing.assert_array_equal(u32(got["linestring_index"]), want["linestring_index"])
    np.testing.assert_array_equal(to_np(got["distance"]), want["distance"])
