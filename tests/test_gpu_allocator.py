"""Calls through a caller's own gbx_allocator: memory aligned to 16 bytes only
(what the interface asks for), and pools with little room.  Results against
numpy, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from cudf_b200 import Column, GroupBy, GroupByRequest, Table
from cudf_b200 import _lib
from cudf_b200 import aggregation as agg
from cudf_b200 import join as J
from cudf_b200._abi import Status, Strategy
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


class TightAllocator(TorchAllocator):
    """Refuses a request beyond `largest` bytes, or one that takes the live bytes beyond `room`."""

    def __init__(self, largest, room=1 << 62):
        super().__init__()
        self.largest, self.room = largest, room

    def _allocate(self, ctx, nbytes, stream):
        if int(nbytes) > self.largest or self.current + int(nbytes) > self.room:
            return None
        return super()._allocate(ctx, nbytes, stream)


def _sums(keys, allocator):
    """{key: rows} of a groupby over the key column, through the allocator."""
    n = len(keys)
    column = Column.from_strings(keys) if isinstance(keys, list) else T.device_column(HostCol(keys))
    gk, res = GroupBy(Table([column])).aggregate(
        [GroupByRequest(T.device_column(HostCol(np.ones(n, dtype=np.int64))), [agg.sum(), agg.median()])],
        allocator=allocator)
    cols = res[0].columns()
    assert np.all(cols[1].to_numpy()[0] == 1.0)
    return dict(zip(gk.columns()[0].to_numpy()[0].tolist(), cols[0].to_numpy()[0].tolist()))


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


@pytest.mark.parametrize("strings", [False, True], ids=["int64", "string"])
def test_a_small_call_asks_for_little(strings):
    """A 100-row call takes kilobytes (a table of 1,024 slots is the most of it), not a block of megabytes."""
    k = np.arange(100, dtype=np.int64) % 7
    want = {int(i): int((k == i).sum()) for i in range(7)}
    if strings:
        k = [f"key {i}" for i in k]
        want = {f"key {i}": n for i, n in want.items()}
    pool = TightAllocator(256 << 10, 512 << 10)
    assert _sums(k, pool) == want
    assert pool.peak <= 256 << 10


def test_a_small_join_asks_for_little():
    left, right = np.arange(100, dtype=np.int64), np.arange(50, dtype=np.int64)
    pool = TightAllocator(64 << 10)
    got = J.inner_join(Table([T.device_column(HostCol(left))]), Table([T.device_column(HostCol(right))]), allocator=pool)
    assert _pairs(got) == [(i, i) for i in range(50)]
    assert pool.peak <= 64 << 10


def test_buffers_that_do_not_fit_in_one_piece_come_one_by_one():
    """20,000 rows: the sample's buffers together are 1.5 MB, the largest of them 1 MB."""
    k = np.arange(20_000, dtype=np.int64) % 100
    assert _sums(k, TightAllocator(1 << 20)) == {i: 200 for i in range(100)}


@pytest.mark.parametrize("join", [J.inner_join, J.left_join, J.full_join], ids=["inner", "left", "full"])
def test_join_where_the_packed_table_has_no_room(join):
    """100,000 build rows: 4 MB of packed slots against 1 MB of row indices."""
    rng = np.random.default_rng(9)
    left, right = np.arange(150_000, dtype=np.int64)[::-1].copy(), rng.permutation(100_000).astype(np.int64)
    pool = TightAllocator(2 << 20)
    got = join(Table([T.device_column(HostCol(left))]), Table([T.device_column(HostCol(right))]), allocator=pool)
    where = np.argsort(right)
    want = [(i, int(where[k])) for i, k in enumerate(left) if k < 100_000]
    if join is not J.inner_join:
        want += [(i, J.JOIN_NONE) for i, k in enumerate(left) if k >= 100_000]
    assert _pairs(got) == sorted(want)


@pytest.mark.parametrize("room", [48 << 10, 100 << 10, 300 << 10, 1 << 20])
def test_a_join_in_a_pool_of_a_few_buffers(room):
    """A pool too small for the shared allocation still serves what fits buffer by buffer, or says that it cannot."""
    left, right = np.arange(2000, dtype=np.int64), np.arange(1000, dtype=np.int64)
    pool = TightAllocator(room, room)
    tables = [Table([T.device_column(HostCol(x))]) for x in (left, right)]
    try:
        got = J.inner_join(*tables, allocator=pool)
    except _lib.GbxError as e:
        assert e.status == Status.ERR_ALLOC and room < 100 << 10
    else:
        assert _pairs(got) == [(i, i) for i in range(1000)]


@pytest.mark.parametrize("columns,groups,hot", [(1, 20_000, 0.0), (5, 12_000, 0.1), (5, 1000, 0.0)],
                         ids=["bucketed", "one_run_an_sm", "skewed"])
def test_bucketed_calls_where_the_copies_have_no_room(columns, groups, hot):
    """4.2M rows: copies of 33 MB a column, against a pool that gives 8 MB at a time."""
    rng = np.random.default_rng(groups)
    n = 4_200_000
    k = rng.integers(0, groups, n)
    k[rng.random(n) < hot] = 3
    vals = [rng.integers(-50, 50, n).astype(np.float64) for _ in range(columns)]
    valid = [rng.random(n) >= 0.1 for _ in vals]
    gb = GroupBy(Table([T.device_column(HostCol(k.astype(np.int64)))]))
    reqs = [GroupByRequest(T.device_column(HostCol(v, ok)), [agg.sum(), agg.count(), agg.mean()])
            for v, ok in zip(vals, valid)]
    free = gb.aggregate(reqs)
    assert gb.last_stats()["strategy"] == Strategy.BUCKETED
    tight = gb.aggregate(reqs, allocator=TightAllocator(8 << 20))
    assert gb.last_stats()["strategy"] != Strategy.BUCKETED
    for gk, res in (free, tight):
        key = gk.columns()[0].to_numpy()[0]
        assert np.array_equal(np.sort(key), np.unique(k))
        for v, ok, t in zip(vals, valid, res):
            want = np.bincount(k[ok], weights=v[ok], minlength=groups)  # whole numbers: exact in any order
            assert np.array_equal(t.columns()[0].to_numpy()[0], want[key])
            assert np.array_equal(t.columns()[1].to_numpy()[0], np.bincount(k[ok], minlength=groups)[key])
