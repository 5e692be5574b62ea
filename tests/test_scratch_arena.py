"""The scratch arena of a one-shot call: the memory a call takes from its
caller's allocator is given back, its outputs are blocks of their own, and a
caller whose memory holds the buffers but no slab gets the same result."""

import numpy as np
import pytest
import torch

import cuspatial_gb300 as cs
from cuspatial_gb300 import _lib, api
from oracle import oracle as O

from helpers import assert_tree_equal

pytestmark = pytest.mark.gpu

ARGS = (0.0, 50.0, 0.0, 50.0, 50.0 / 32, 5, 16)


class _Counting(_lib.TorchAllocator):
    made = []

    def __init__(self, *a, **k):
        super().__init__(*a, **k)
        self.made.append(self)

    def _allocate(self, ctx, nbytes, stream):
        if self.limit is not None and nbytes > self.limit:
            return None
        return super()._allocate(ctx, nbytes, stream)


@pytest.mark.parametrize("limit", [None, 1 << 20])
@pytest.mark.parametrize("n", [1, 1003, 60_000])
def test_outputs_are_own_blocks_and_scratch_goes_back(monkeypatch, n, limit):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 50, (2, n))
    _Counting.limit, _Counting.made = limit, []
    monkeypatch.setattr(api._lib, "TorchAllocator", _Counting)
    pi, tree = cs.quadtree_on_points(cs.GeoSeries.from_points(x, y), *ARGS)
    torch.cuda.synchronize()
    (a,) = _Counting.made
    assert not a.blocks and a.in_use == 0  # all scratch returned, outputs adopted
    # outputs written by later calls' scratch would show here
    cs.quadtree_on_points(cs.GeoSeries.from_points(y, x), *ARGS)
    assert_tree_equal(pi, tree, *O.quadtree_on_points(x, y, *ARGS))
