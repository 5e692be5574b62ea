"""The filtered nearest call over many points with some leaves that its listing cannot
take (more segments near them than it lists), holding few points or many, so that
either exact kernel takes them: against the oracle bit for bit."""

import numpy as np
import pytest

from test_nearest_far_segments import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowd", [1, 200, 3900, 4300, 12_000])
def test_leaves_with_many_segments_near_them(crowd):
    rng = np.random.default_rng(crowd)
    n, count, dense, vertices = 9000, 30, 70, 13
    lx, ly = rng.uniform(0, 40, (2, (count + dense) * vertices))
    part = np.arange(0, (count + dense + 1) * vertices, vertices, dtype=np.int32)
    # 840 segments in a corner of one leaf, 384 can be listed
    a = part[count]
    lx[a:], ly[a:] = 21.0 + 0.5 * rng.random(len(lx) - a), 21.0 + 0.5 * rng.random(len(lx) - a)
    x, y = rng.uniform(0, 40, (2, n + crowd))
    x[n:], y[n:] = 20.9 + 0.7 * rng.random(crowd), 20.9 + 0.7 * rng.random(crowd)
    j = rng.integers(0, len(lx), n + crowd)
    on = rng.random(n + crowd) < 0.02
    x, y = np.where(on, lx[j], x), np.where(on, ly[j], y)
    check(x, y, lx, ly, part, "filtered", 200)
