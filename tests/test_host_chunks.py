"""Host points and host rows where the number of copied chunks changes, against the
device entry points (exactly)."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300 import datasets as D
from helpers import gpu_points, gpu_polygons

pytestmark = pytest.mark.gpu

M = 1 << 20  # one chunk below 2 Mi points, two from there, then one for every 4 Mi


@pytest.mark.parametrize("n", [2 * M - 1, 2 * M, 12 * M - 1, 12 * M, 21 * M + 7])
def test_point_chunks(n):
    rng = np.random.default_rng(n)
    # whole numbers: equal keys in every chunk, whose order the merge has to keep
    x, y = (torch.from_numpy(rng.integers(0, 1001, n).astype(np.float32)).pin_memory()
            for _ in range(2))
    args = (0.0, 1000.0, 0.0, 1000.0, 1000.0 / (1 << 9), 9, 200)
    pts, pi, t, xy = cs.quadtree_on_points_host(x, y, *args, ordered=True)
    assert torch.equal(pts.points.x.cpu(), x) and torch.equal(pts.points.y.cpu(), y)
    pi2, t2 = cs.quadtree_on_points(cs.GeoSeries.from_points(x.cuda(), y.cuda()), *args)
    assert torch.equal(pi, pi2)
    for k in t2:
        assert torch.equal(t[k], t2[k]), k
    xy = xy.reshape(-1, 2)
    at = pi.cpu().long()
    assert torch.equal(xy[:, 0].cpu(), x[at]) and torch.equal(xy[:, 1].cpu(), y[at])


@pytest.mark.parametrize("method", ["exact", "filtered"])
def test_row_chunks(method):
    w = D.precision_at_scale(n_points=2_000_000, n_polygons=40_000, extent=4000.0,
                             max_vertices=32)
    args = (w.x_min, w.x_max, w.y_min, w.y_max, w.scale, w.max_depth)
    pts, polys = gpu_points(w), gpu_polygons(w.polygons)
    pi, t = cs.quadtree_on_points(pts, *args, 32)
    j = cs.join_quadtree_and_bounding_boxes(t, cs.polygon_bounding_boxes(polys), *args)
    assert int(j["bbox_offset"].numel()) >= 3 << 18
    for k in ((1 << 19) - 1, 1 << 19, 3 << 18, int(j["bbox_offset"].numel())):  # 1, 2, 3 chunks
        part = {c: j[c][:k] for c in ("bbox_offset", "quad_offset")}
        want = cs.quadtree_point_in_polygon(part, t, pi, pts, polys, method=method)
        m = int(want["polygon_index"].numel())
        out = [torch.full((m + 3,), -1, dtype=torch.int32, pin_memory=True) for _ in range(2)]
        assert cs.quadtree_point_in_polygon_host(part, t, pi, pts, polys, *out,
                                                 method=method) == m
        for o, c in zip(out, ("polygon_index", "point_index")):
            assert torch.equal(o[:m], want[c].cpu().view(torch.int32))
            assert o[m:].tolist() == [-1] * 3
        small = torch.empty(m - 1, dtype=torch.int32)  # too few rows: the count comes back
        with pytest.raises(cs.HostRowsTooFew) as e:
            cs.quadtree_point_in_polygon_host(part, t, pi, pts, polys, small, small.clone(),
                                              method=method)
        assert e.value.rows == m
