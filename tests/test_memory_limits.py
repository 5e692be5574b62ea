"""Calls whose memory is limited: the faster ways of a call (wider appends and the
node table of the box join, float32 bounds, the grid of cells, boxes of segments)
are taken where there is room, and where there is not the call needs no more than
without them."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300 import _lib, api

from helpers import gpu_polygons
from test_pip_large_offsets import layer

pytestmark = pytest.mark.gpu

KB = 1 << 10


@pytest.fixture
def budget(monkeypatch):
    class Limited(_lib.TorchAllocator):
        limit = last = None

        def __init__(self, *a, **k):
            super().__init__(*a, **k)
            self.budget = Limited.limit
            Limited.last = self

    monkeypatch.setattr(api._lib, "TorchAllocator", Limited)
    return Limited


def _points(n, seed, ext=20.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, y = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * ext
            for _ in range(2))
    return cs.GeoSeries.from_points(x, y)


def _boxes(rng, count, lo, hi):
    c, h = rng.uniform(2, 18, (2, count)), rng.uniform(lo, hi, (2, count))
    return {k: torch.from_numpy(v).cuda() for k, v in
            zip(("minx", "miny", "maxx", "maxy"), (*(c - h), *(c + h)))}


def _same(a, b):
    for k in a:
        assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("n,max_size,boxes,half", [
    (200_000, 16, 1, 3.0),  # all pairs of few boxes are appended where there is room
    (200_000, 16, 40, 0.5),
    (16_700_000, 32, 24, 4.5),  # more pairs than that: the write pass, with its table
])
def test_join_in_eight_words_a_pair(budget, n, max_size, boxes, half):
    rng = np.random.default_rng(boxes)
    args = (0.0, 20.0, 0.0, 20.0, 20.0 / 2 ** 12, 12)
    _, tree = cs.quadtree_on_points(_points(n, 1), *args, max_size)
    bb = _boxes(rng, boxes, half, half)
    want = cs.join_quadtree_and_bounding_boxes(tree, bb, *args)
    k = want["bbox_offset"].numel()
    assert n < 10 ** 6 or (k > 4 << 20 and n <= 4 * k)
    # key, box, node and permutation twice or once each, the sort's counts
    budget.limit = 33 * k + 512 * boxes + 64 * KB
    _same(want, cs.join_quadtree_and_bounding_boxes(tree, bb, *args))
    assert budget.last.peak <= budget.limit


def _least(budget, call, most):
    """The smallest limit that `call` does its work in, to a hundredth."""
    low, high = 0, most
    while high - low > max(4 * KB, high // 100):
        mid = (low + high) // 2
        budget.limit = mid
        try:
            call()
            high = mid
        except MemoryError:
            low = mid
    budget.limit = None
    return high


def test_bounds_and_cells_do_not_raise_what_a_call_needs(budget):
    # one point more takes the faster way where there is room
    P = layer(np.random.default_rng(3), 31, 1.0)
    polys, need = gpu_polygons(P), {}
    for n in (65_535, 65_536):
        pts = _points(n, 2)
        args = (0.0, 20.0, 0.0, 20.0, 20.0 / 2 ** 8, 8)
        pi, tree = cs.quadtree_on_points(pts, *args, 32)
        pairs = cs.join_quadtree_and_bounding_boxes(tree, cs.polygon_bounding_boxes(polys), *args)

        def join():
            return cs.quadtree_point_in_polygon(pairs, tree, pi, pts, polys, method="exact")

        def mask():
            return cs.point_in_polygon_bitmask(pts, polys, "exact")

        rows, bits = join(), mask()
        need[n] = [_least(budget, c, 256 << 20) for c in (join, mask)]
        budget.limit = need[n][0]
        _same(rows, join())
        budget.limit = need[n][1]
        assert torch.equal(bits, mask())
        budget.limit = None
    for few, many in zip(*need.values()):
        assert many <= few * 1.02 + 16 * KB


@pytest.mark.parametrize("method", ["exact", "filtered"])
@pytest.mark.parametrize("n", [3000, 60_000])
def test_nearest_without_boxes(budget, n, method):
    rng = np.random.default_rng(4)
    count, vertices = 300, 61
    steps = rng.uniform(-0.2, 0.2, (2, count, vertices))
    lx, ly = (rng.uniform(0, 20, (2, count, 1)) + np.cumsum(steps, 2)).reshape(2, -1)
    off = np.arange(count + 1, dtype=np.int32)
    lines = cs.GeoSeries.from_linestrings_xy(np.stack([lx, ly], 1).reshape(-1), off * vertices,
                                             off)
    args = (0.0, 20.0, 0.0, 20.0, 20.0 / 2 ** 7, 7)
    pts = _points(n, 5)
    pi, tree = cs.quadtree_on_points(pts, *args, 32)
    pairs = cs.join_quadtree_and_bounding_boxes(tree, cs.linestring_bounding_boxes(lines, 4.0),
                                                *args)

    def call():
        return cs.quadtree_point_to_nearest_linestring(pairs, tree, pi, pts, lines, method=method)

    want, k = call(), pairs["bbox_offset"].numel()
    # exact: the groups' starts; filtered: frames of 56 bytes a group, points and
    # segments in float32, the linestrings' records and their boxes
    exact = 4 * k + 32 * KB
    budget.limit = exact if method == "exact" else (exact + 64 * k + 8 * n +
                                                    20 * lx.size + 256 * count)
    _same(want, call())
