"""Nearest linestrings where a segment's distance is not a number although its
start is finite: the other end NaN or infinite, so far away that the squares
overflow, or so near that they underflow.  Such a segment contributes nothing to
its linestring's distance, and its start bounds nothing.  Both kernels of the
exact method (a warp per point up to 4096 points, a lane per point above) and
the groups the filtered method leaves to them, against the oracle bit for bit."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import to_np, u32

pytestmark = pytest.mark.gpu


def check(x, y, lx, ly, part, method, max_size, ext=40.0):
    """Every leaf against every linestring, in the reference's order."""
    args = (0.0, ext, 0.0, ext, ext / 16, 4)
    pts = cs.GeoSeries.from_points(x, y)
    xy = np.stack([lx, ly], 1).reshape(-1)
    nl = len(part) - 1
    ls = cs.GeoSeries.from_linestrings_xy(xy, part, np.arange(nl + 1, dtype=np.int32))
    pi, tree = cs.quadtree_on_points(pts, *args, max_size)
    opi, ot = O.quadtree_on_points(x, y, *args, max_size)
    q = np.flatnonzero(~ot["is_internal_node"])
    q = q[np.argsort(ot["offset"][q], kind="stable")]
    pairs = {"bbox_offset": np.tile(np.arange(nl, dtype=np.int32), len(q)),
             "quad_offset": np.repeat(q.astype(np.int32), nl)}
    gp = {k: torch.from_numpy(v).cuda() for k, v in pairs.items()}
    got = cs.quadtree_point_to_nearest_linestring(gp, tree, pi, pts, ls, method=method)
    want = O.quadtree_point_to_nearest_linestring(pairs, ot, opi, x, y, part, lx, ly)
    np.testing.assert_array_equal(u32(got["linestring_index"]), want["linestring_index"])
    np.testing.assert_array_equal(to_np(got["distance"]), want["distance"])


def _lines(rng, count, vertices, ext, dtype):
    lx, ly = rng.uniform(0, ext, (2, count * vertices)).astype(dtype)
    return lx, ly, np.arange(0, (count + 1) * vertices, vertices, dtype=np.int32)


@pytest.mark.parametrize("dtype,method", [(np.float64, "exact"), (np.float64, "filtered"),
                                          (np.float32, "exact")])
@pytest.mark.parametrize("n,max_size", [(1, 8), (600, 40), (4096, 300), (4097, 300), (9000, 700)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, "far", "near"])
def test_segments_without_a_distance(dtype, method, n, max_size, bad):
    # linestring p has its p-th vertex among the points and no number on either
    # side of it, its other vertices are the farthest: not the nearest, whichever
    # of its two chunks of 8 segments and a part of one that vertex starts
    rng = np.random.default_rng([n, max_size])
    vertices, honest = 19, 6
    lx, ly, part = _lines(rng, vertices + honest, vertices, 40.0, dtype)
    lures = part[vertices]
    lx[:lures], ly[:lures] = 30 + lx[:lures] / 8, 30 + ly[:lures] / 8
    lx[lures:], ly[lures:] = 8 + lx[lures:] / 8, 8 + ly[lures:] / 8
    f32 = dtype == np.float32
    tiny, far = (1e-24, 1e20) if f32 else (1e-170, 1e160)
    for p in range(vertices):
        at = {0: rng.uniform(0, 1)}
        if bad == "near":  # segments so short that their squares are zero
            at = {-2: np.nan, -1: -tiny, 0: 0.0, 1: tiny, 2: np.nan}
        elif bad == "far":  # so long that the points beyond its start see infinity
            at.update({-1: np.nan, 1: far})
        else:
            at.update({-1: bad, 1: bad})
        for d, v in at.items():
            if 0 <= p + d < vertices:
                lx[part[p] + p + d] = ly[part[p] + p + d] = v
    x, y = rng.uniform(0, 1, (2, n)).astype(dtype)
    check(x, y, lx, ly, part, method, max_size, ext=1.0)


@pytest.mark.parametrize("dtype,method", [(np.float64, "exact"), (np.float64, "filtered"),
                                          (np.float32, "exact")])
def test_only_the_bounding_linestring_is_near(dtype, method):
    # A starts beside the point and goes on to a vertex that is not a number, its
    # other segments are far; B is the winner, beyond A's start
    for n in (1, 5000):
        x, y = np.full(n, 1.0, dtype), np.zeros(n, dtype)
        lx = np.array([0, np.nan, 100, 101, 10, 10], dtype)
        ly = np.array([0, np.nan, 100, 100, 0, 1], dtype)
        check(x, y, lx, ly, np.array([0, 4, 6], np.int32), method, n)


@pytest.mark.parametrize("method", ["exact", "filtered"])
@pytest.mark.parametrize("n,max_size,dense", [(4096, 300, False), (4097, 300, False),
                                              (30_000, 2000, False), (6000, 3000, True)])
def test_adversarial_points_beyond_a_warp_per_point(method, n, max_size, dense):
    # zero distances (passed over), repeated linestrings (ties by id), leaves of
    # more than 256 points; dense: more segments near a leaf than the filtered
    # method lists, so that its groups are left to the exact kernels
    rng = np.random.default_rng([n, max_size])
    count, vertices = (60, 40) if dense else (20, 19)
    lx, ly, part = _lines(rng, count, vertices, 40.0, np.float64)
    for k in range(3, count, 7):
        a, b = part[k], part[k - 1]
        lx[a:a + vertices], ly[a:a + vertices] = lx[b:b + vertices], ly[b:b + vertices]
    x, y = rng.uniform(0, 40, (2, n))
    j = rng.integers(0, len(lx), n)
    on = rng.random(n) < 0.2
    x, y = np.where(on, lx[j], x), np.where(on, ly[j], y)
    check(x, y, lx, ly, part, method, max_size)
