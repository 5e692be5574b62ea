"""Polygons whose height spans a few float32 steps of their y: the rises that size the
slab index are lost to float32, the number of slab entries must keep to the arrays all
the same.  Joins, the bitmask call and a batched plan against the oracle; the entries
that the slab count alone would give are counted on the host to be beyond the arrays."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300.batched import BatchedPointInPolygon
from cuspatial_gb300.datasets import Polygons
from oracle import oracle as O

from helpers import gpu_polygons, to_np
from test_pip_large_offsets import join, join_oracle

AT = 2.0 ** 25  # float32 steps of 4


def zigzag(rng, count, vertices, top):
    """Fans of spikes: nearly all of the rise lies within one float32 step of a polygon
    that is top / 4 of them high."""
    x, y, ro = [], [], [0]
    for _ in range(count):
        c = AT + 4.0 * rng.integers(0, 4, 2)
        k = 2 * vertices
        vx = c[0] + 0.001 + 3.9 * np.arange(k) / k
        vy = c[1] + np.where(np.arange(k) % 2, 0.1, 3.8) + 0.05 * rng.random(k)
        # the way back above, over the other steps
        x.append(np.concatenate([vx, [c[0] + 3.95, c[0], vx[0]]]))
        y.append(np.concatenate([vy, [c[1] + top, c[1] + top, vy[0]]]))
        ro.append(ro[-1] + k + 3)
    i = np.arange(count + 1, dtype=np.int32)
    return Polygons(np.concatenate(x), np.concatenate(y), np.array(ro, np.int32), i, i)


@pytest.mark.parametrize("top,vertices", [(6.0, 100), (400.0, 3000)])
def test_truncated_rises_would_exceed_the_arrays(top, vertices):
    P = zigzag(np.random.default_rng(1), 6, vertices, top)
    for density in (2.0, 8.0):
        entries = 0.0
        for p in range(6):
            y = P.y[P.ring_offset[p]:P.ring_offset[p + 1]]
            nv, height = len(y), y.max() - y.min()
            step = np.floor(y / 4.0) * 4.0  # as float32 cut toward zero
            s = density * nv * height / np.abs(np.diff(step)).sum()
            slabs = int(max(1.0, min(s, 0.5 * density * nv, 4096)))
            entries += np.abs(np.diff(y)).sum() * slabs / height
        assert entries > 2 * (density + 2) * len(P.y)


@pytest.mark.gpu
@pytest.mark.parametrize("count,vertices,top", [(1, 4, 6.0), (1, 100, 6.0), (25, 100, 6.0),
                                                (7, 3000, 6.0), (7, 3000, 400.0),
                                                (25, 300, 270.0)])
@pytest.mark.parametrize("n,method", [(3000, "exact"), (70_000, "exact"), (3000, "filtered"),
                                      (140_000, "filtered")])
def test_against_oracle(count, vertices, top, n, method):
    rng = np.random.default_rng([count, vertices])
    P = zigzag(rng, count, vertices, top)
    if n * len(P.x) > 2e9:
        n = 5000
    x, y = AT + rng.uniform(-1, 23, (2, n))
    y = np.where(rng.random(n) < 0.2, AT + rng.uniform(-1, top + 20, n), y)
    j = rng.integers(0, len(P.x), n)
    on = rng.random(n) < 0.1
    x, y = np.where(on, P.x[j], x), np.where(rng.random(n) < 0.1, P.y[j], y)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P)
    got = cs.point_in_polygon_bitmask(pts, polys, method)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y)
    np.testing.assert_array_equal(to_np(got).view(np.uint32), want.view(np.uint32))
    a = (AT - 2, AT + top + 24, 5, 100)
    got, want = join(x, y, P, *a, method), join_oracle(x, y, P, *a)
    for k in ("polygon_index", "point_index"):
        np.testing.assert_array_equal(to_np(got[k]), want[k].astype(np.int32))
    if n > 5000:
        return
    for ordered in (False, True):
        with BatchedPointInPolygon(
                torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), [0, n], polys, [0, count],
                [(AT - 2, a[1], AT - 2, a[1], (a[1] - AT + 2) / 32, 5, 100)], method=method,
                ordered_index=ordered) as plan:
            _, polygon, point = plan.run().rows()
            for g, k in ((polygon, "polygon_index"), (point, "point_index")):
                np.testing.assert_array_equal(to_np(g), want[k].astype(np.int32))
