"""The memory a batched plan keeps beside its own buffers."""

import numpy as np
import pytest
import torch

from cuspatial_gb300 import _lib
from cuspatial_gb300.batched import BatchedPointInPolygon

from helpers import gpu_polygons, to_np
from test_pip_large_offsets import layer

pytestmark = pytest.mark.gpu


def test_small_plan_keeps_little():
    P = layer(np.random.default_rng(6), 3, 1.0)
    g = torch.Generator(device="cuda").manual_seed(7)
    x, y = (torch.rand(1000, generator=g, device="cuda", dtype=torch.float64) * 20
            for _ in range(2))
    with BatchedPointInPolygon(x, y, [0, 1000], gpu_polygons(P), [0, 3],
                               [(0.0, 20.0, 0.0, 20.0, 20.0 / 32, 5, 32)]) as plan:
        (alloc,) = [v for v in vars(plan).values() if isinstance(v, _lib.TorchAllocator)]
        plan.run()
        offsets, polygon, point = (to_np(t).copy() for t in plan.rows())
        # a first slab of 1 MiB on each of its two streams and the rows
        assert alloc.in_use <= (2 << 20) + (256 << 10)
    assert alloc.in_use == 0
    assert offsets[-1] == len(polygon) == len(point) > 0
