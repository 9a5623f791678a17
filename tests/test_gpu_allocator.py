"""Calls through a caller's own gbx_allocator: memory aligned to 16 bytes only
(what the interface asks for).  Results against numpy, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from cudf_b200 import Table
from cudf_b200 import join as J
from cudf_b200.groupby import TorchAllocator
from oracle.oracle import HostCol
from tests import gbx_testing as T

pytestmark = pytest.mark.gpu


class OffsetAllocator(TorchAllocator):
    """Memory that starts `offset` bytes into its block."""

    def __init__(self, offset):
        super().__init__()
        self.offset = offset

    def _allocate(self, ctx, nbytes, stream):
        p = super()._allocate(ctx, int(nbytes) + self.offset, stream)
        if p is None:
            return None
        block = self.live.pop(p)
        self.live[p + self.offset] = block[self.offset:]
        return p + self.offset


def _pairs(cols):
    return sorted(zip(*(c.to_numpy()[0].tolist() for c in cols)))


@pytest.mark.parametrize("offset", [16, 32, 48])
@pytest.mark.parametrize("rows", [700, 300_000])  # slots carved from a shared block, and in a block of their own
def test_packed_join_on_memory_aligned_to_16_bytes(rows, offset):
    rng = np.random.default_rng(rows)
    left, right = rng.integers(0, 2 * rows, 3000), rng.permutation(rows)
    cols = J.inner_join(Table([T.device_column(HostCol(left.astype(np.int64)))]),
                        Table([T.device_column(HostCol(right.astype(np.int64)))]), allocator=OffsetAllocator(offset))
    where = {int(k): i for i, k in enumerate(right)}
    assert _pairs(cols) == [(i, where[int(k)]) for i, k in enumerate(left) if int(k) in where]
