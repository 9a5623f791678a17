"""Joins whose key packs into one 64-bit word (gbx_join_packed.cu) against the
join oracle: unique and repeated build keys, row counts around the 2,048-row
probe tile, the all-ones key (the table's empty word), several key layouts,
nulls and sliced columns.  Pairs are compared bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from cudf_b200 import Table
from cudf_b200 import join as J
from cudf_b200._abi import JoinKind, NullEquality
from oracle.oracle import HostCol
from tests import gbx_testing as T
from tests.test_gpu_join import KINDS, _check

pytestmark = pytest.mark.gpu


def _keys(layout, idx, rng):
    """Key columns of the key numbers `idx`; number 0 is all ones where the layout allows it."""
    if layout == "int64":
        return [HostCol((idx.astype(np.int64) * 982_451_653) - 1)]
    if layout == "int32":
        return [HostCol(idx.astype(np.int32) - 1)]
    if layout == "int32_int16_nulls":
        valid = (idx % 7) != 3  # a null key column, the same for equal numbers
        return [HostCol(idx.astype(np.int32) * 77), HostCol((idx % 1000).astype(np.int16), valid)]
    v = (idx - 5).astype(np.float64) * 0.5
    v[idx == 5] = np.where(rng.random(int((idx == 5).sum())) < 0.5, -0.0, 0.0)
    v[idx == 9] = np.nan
    return [HostCol(v)]


@pytest.mark.parametrize("layout", ["int64", "int32", "int32_int16_nulls", "float64"])
@pytest.mark.parametrize("repeated", [False, True], ids=["unique", "repeated"])
@pytest.mark.parametrize("nl,nr", [(1, 1), (2047, 60), (2048, 700), (2049, 3000), (6145, 1500)])
def test_packed_join_matches_oracle(layout, repeated, nl, nr):
    rng = np.random.default_rng(nl * 7 + nr)
    right = rng.integers(0, max(1, nr // 3), nr) if repeated else rng.permutation(nr)
    left = rng.integers(0, max(2, nr + nr // 4), nl)
    left[0] = 0
    for kind in KINDS:
        for nulls in (NullEquality.EQUAL, NullEquality.UNEQUAL):
            _check(_keys(layout, left, rng), _keys(layout, right, rng), nulls, kind)


def test_packed_join_of_sliced_columns():
    rng = np.random.default_rng(5)
    a, b = rng.integers(0, 300, 5000), rng.permutation(400)
    left = Table([T.device_column(HostCol(a.astype(np.int64))).slice(13, 4111)])
    right = Table([T.device_column(HostCol(b.astype(np.int64))).slice(7, 390)])
    li, ri = (c.to_numpy()[0] for c in J.inner_join(left, right))
    where = {int(k): i for i, k in enumerate(b[7:390])}
    want = [(i, where[int(k)]) for i, k in enumerate(a[13:4111]) if int(k) in where]
    assert sorted(zip(li.tolist(), ri.tolist())) == want


@pytest.mark.parametrize("nl,nr,card", [(1, 1, 1), (31, 4000, 3), (2048, 2500, 900), (2100, 3000, 30), (4097, 20_000, 50)])
def test_repeated_keys_come_in_left_row_order(nl, nr, card):
    """Each left row's pairs follow one another in row order; many outputs share a tile among several blocks."""
    rng = np.random.default_rng(nl + nr)
    left, right = rng.integers(0, card + 1, nl), rng.integers(0, card, nr)
    right[0] = right[-1] = 0  # a repeated key
    cols = [Table([T.device_column(HostCol(x.astype(np.int64)))]) for x in (left, right)]
    li, ri = (c.to_numpy()[0] for c in J.left_join(*cols))
    counts = np.bincount(right, minlength=card + 1)
    assert np.array_equal(li, np.repeat(np.arange(nl), np.maximum(counts[left], 1)))
    order = np.argsort(right, kind="stable")
    first = np.cumsum(counts) - counts
    want = np.concatenate([order[first[k]:first[k] + counts[k]] if counts[k] else [J.JOIN_NONE] for k in left])
    assert np.array_equal(ri[np.lexsort((ri, li))], want)


@pytest.mark.parametrize("join", [J.inner_join, J.left_join, J.full_join], ids=["inner", "left", "full"])
@pytest.mark.parametrize("repeated", [False, True], ids=["unique", "repeated"])
@pytest.mark.parametrize("nl", [190_000, 230_000])
def test_both_sides_of_the_line_for_tables_beyond_l2(nl, repeated, join):
    """3.2M build rows (134 MB of slots): one probe row to 16 build rows is where the packed table begins to pay."""
    rng = np.random.default_rng(nl)
    nr = 3_200_000
    right = rng.integers(0, nr, nr) if repeated else rng.permutation(nr)
    left = rng.integers(0, nr + nr // 8, nl)
    cols = [Table([T.device_column(HostCol(x.astype(np.int64)))]) for x in (left, right)]
    li, ri = (c.to_numpy()[0].astype(np.int64) for c in join(*cols))
    counts = np.bincount(right, minlength=nr + nr // 8)
    order = np.argsort(right, kind="stable")
    first = np.cumsum(counts) - counts
    c = counts[left]
    at = np.repeat(np.arange(nl), c)
    want_l = at
    want_r = order[first[left][at] + (np.arange(len(at)) - np.repeat(np.cumsum(c) - c, c))]
    if join is not J.inner_join:
        none = np.flatnonzero(c == 0)
        want_l, want_r = np.concatenate([want_l, none]), np.concatenate([want_r, np.full(len(none), J.JOIN_NONE)])
    if join is J.full_join:
        rest = np.flatnonzero(~np.isin(right, left))
        want_l, want_r = np.concatenate([want_l, np.full(len(rest), J.JOIN_NONE)]), np.concatenate([want_r, rest])
    got, want = np.lexsort((ri, li)), np.lexsort((want_r, want_l))
    assert np.array_equal(li[got], want_l[want]) and np.array_equal(ri[got], want_r[want])
