"""pairwise_point_in_polygon's walk over runs of 32 pairs, rings and vertices:
sizes at the edges of those runs, several rings per polygon, empty rings and
polygons, coordinates far from the origin and at zero, against the oracle
(exactly: the results are flags).  split_f32 (csrc/f32_split.cuh) is checked
on the host against exact rational arithmetic."""

import ctypes
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import cuspatial_gb300 as cs
from oracle import oracle as O

from helpers import gpu_polygons, to_np

HERE = os.path.dirname(os.path.abspath(__file__))


def _rings(rng, n, sizes, max_rings, scale, at):
    """n polygons of 0..max_rings star rings with sizes drawn from `sizes`,
    radius about `scale`, centred near `at`."""
    from cuspatial_gb300.datasets import Polygons
    x, y, ro, po = [], [], [0], [0]
    px, py = np.empty(n), np.empty(n)
    for i in range(n):
        c = at + rng.uniform(-5, 5, 2) * scale
        for r in range(rng.integers(0 if n > 1 else 1, max_rings + 1)):
            k = int(rng.choice(sizes))
            a = np.sort(rng.uniform(0, 2 * np.pi, k))
            d = scale * rng.uniform(0.4, 1.0, k) * (1.0 if r == 0 else 0.4)
            vx, vy = c[0] + d * np.cos(a), c[1] + d * np.sin(a)
            if k and rng.random() < 0.7:  # closed; others are left open
                vx, vy = np.append(vx, vx[0]), np.append(vy, vy[0])
            x.append(vx)
            y.append(vy)
            ro.append(ro[-1] + len(vx))
        po.append(len(ro) - 1)
        px[i], py[i] = c + rng.uniform(-1, 1, 2) * scale
        own = [v for v in range(po[-2], po[-1]) if ro[v + 1] > ro[v]]
        if own and rng.random() < 0.3:  # on a vertex, or level with one
            v = int(rng.choice(own))
            j = int(rng.integers(0, ro[v + 1] - ro[v]))
            py[i] = y[v][j]
            if rng.random() < 0.6:
                px[i] = x[v][j]
    cat = lambda v: np.concatenate(v) if v else np.zeros(0)  # noqa: E731
    P = Polygons(cat(x), cat(y), np.array(ro, np.int32), np.array(po, np.int32),
                 np.arange(n + 1, dtype=np.int32))
    return px, py, P


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,sizes,max_rings,scale,at", [
    (1, [3], 1, 1.0, 0.0),
    (31, [0, 1, 2, 3, 4], 3, 1.0, 10.0),
    (33, [31, 32, 33], 2, 10.0, 1e3),
    (64, [4], 40, 1.0, -50.0),
    (200, [5, 63, 64, 65, 400], 2, 1e-3, 1e6),
    (500, [7, 3000], 1, 1e5, -1e7),
    (9000, [4, 9], 2, 1.0, 0.0),
    (40000, [3, 5, 70], 2, 20.0, 1e3),
    (300000, [3, 4], 3, 1e-4, 120.0),
])
def test_pairwise_runs_against_oracle(n, sizes, max_rings, scale, at, dtype):
    rng = np.random.default_rng(n)
    x, y, P = _rings(rng, n, sizes, max_rings, scale, at)
    x, y = x.astype(dtype), y.astype(dtype)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x.astype(dtype),
                              P.y.astype(dtype), pairwise=True)
    pts, polys = cs.GeoSeries.from_points(x, y), gpu_polygons(P, dtype)
    for method in ("exact", "filtered"):
        got = to_np(cs.pairwise_point_in_polygon(pts, polys, method))
        np.testing.assert_array_equal(got, want, err_msg=method)


@pytest.mark.gpu
@pytest.mark.parametrize("unit", [1.0, 1e-290, 1e-170, 1e-60, 2.0 ** -100, 1e35, 1e200])
def test_pairwise_magnitudes_against_oracle(unit):
    # squares and triangles with corners and points at multiples of a unit,
    # zero among them: vertical and horizontal edges, points level with
    # corners, products that underflow or overflow
    from cuspatial_gb300.datasets import Polygons
    rng = np.random.default_rng(5)
    n = 400
    k = rng.integers(3, 7, n)
    ro = np.concatenate([[0], np.cumsum(k)]).astype(np.int32)
    px = rng.integers(-2, 3, ro[-1]) * unit
    py = rng.integers(-2, 3, ro[-1]) * unit
    x, y = rng.integers(-4, 5, n) * 0.5 * unit, rng.integers(-4, 5, n) * 0.5 * unit
    ids = np.arange(n + 1, dtype=np.int32)
    P = Polygons(px, py, ro, ids, ids)
    want = O.point_in_polygon(x, y, P.part_offset, P.ring_offset, P.x, P.y, pairwise=True)
    for method in ("exact", "filtered"):
        got = to_np(cs.pairwise_point_in_polygon(cs.GeoSeries.from_points(x, y),
                                                 gpu_polygons(P), method))
        np.testing.assert_array_equal(got, want, err_msg=method)


def test_split_f32_against_rationals(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src, out = tmp_path / "split.cpp", str(tmp_path / "libsplit.so")
    src.write_text('#include <cstddef>\n#include "%s"\n' % os.path.join(
        HERE, "..", "cuspatial_gb300", "csrc", "f32_split.cuh") + '''
extern "C" void split(const double* v, size_t n, float* hi, float* lo, int* ok)
{
  for (size_t i = 0; i < n; ++i) {
    ok[i]                 = cspt::splits_f32(v[i]);
    cspt::F32Pair const p = cspt::split_f32(v[i]);
    hi[i]                 = p.hi;
    lo[i]                 = p.lo;
  }
}
''')
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", str(src), "-o", out],
                   check=True)
    rng = np.random.default_rng(1)
    v = np.concatenate([
        rng.uniform(-1e4, 1e4, 3000), rng.uniform(-1, 1, 1000) * 2.0 ** rng.integers(-110, 110, 1000),
        [0.0, -0.0, np.inf, -np.inf, np.nan, 2.0 ** -100, np.nextafter(2.0 ** -100, 0),
         -2.0 ** 100, np.nextafter(2.0 ** 100, 0), 5e-324, 1.0, np.nextafter(2.0, 0)]])
    hi, lo = np.empty(len(v), np.float32), np.empty(len(v), np.float32)
    ok = np.empty(len(v), np.int32)
    ctypes.CDLL(out).split(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(len(v)),
                           hi.ctypes.data_as(ctypes.c_void_p), lo.ctypes.data_as(ctypes.c_void_p),
                           ok.ctypes.data_as(ctypes.c_void_p))
    with np.errstate(invalid="ignore"):
        covered = np.isfinite(v) & (np.abs(v) >= 2.0 ** -100) & (np.abs(v) < 2.0 ** 100)
    np.testing.assert_array_equal(ok.astype(bool), covered)
    for a, h, l in zip(v[covered], hi[covered], lo[covered]):
        rest = abs(Fraction(float(a))) - abs(Fraction(float(h))) - abs(Fraction(float(l)))
        assert 0 <= rest < Fraction(abs(float(a))) / 2 ** 46
        assert abs(float(l)) < abs(float(a)) * 2.0 ** -23
        assert h * a > 0 and l * a >= 0
