"""The tile-grouping kernel (gbx_tiled.cu) against the oracle where it can go
wrong: row counts around a block, a batch and a tile, one group and groups
beyond a table (listed rows), narrow and wide value types side by side, nulls,
dictionaries and two-word keys.  Tolerances are those of gbx_testing.py."""
from __future__ import annotations

import numpy as np
import pytest

from cudf_b200._abi import Kind, NullPolicy, Strategy
from oracle.oracle import HostCol
from tests import gbx_testing as T

pytestmark = pytest.mark.gpu

ALL = [(k, 1 if k == Kind.VARIANCE else 0) for k in (Kind.SUM, Kind.COUNT_VALID, Kind.COUNT_ALL, Kind.MIN, Kind.MAX,
                                                     Kind.MEAN, Kind.VARIANCE, Kind.SUM_OF_SQUARES, Kind.PRODUCT)]
SIX = [(Kind.SUM, 0), (Kind.COUNT_VALID, 0), (Kind.MIN, 0), (Kind.MAX, 0), (Kind.MEAN, 0), (Kind.VARIANCE, 1)]


@pytest.mark.parametrize("strategy", [Strategy.PRIVATIZED, Strategy.BUCKETED], ids=lambda s: s.name)
@pytest.mark.parametrize("groups", [1, 3, 100, 900, 3000])
@pytest.mark.parametrize("n", [1, 511, 513, 4097, 300_001])
def test_two_channels(n, groups, strategy):
    rng = np.random.default_rng(n + groups)
    k = rng.integers(0, groups, n).astype(np.int64)
    b = rng.standard_normal(n).astype(np.float32)
    b[::97] = np.nan
    T.assert_parity([HostCol(k)], [(HostCol(rng.integers(-10 ** 6, 10 ** 6, n)), SIX),
                                   (HostCol(b, rng.random(n) >= 0.1), SIX)], strategy=strategy)


@pytest.mark.parametrize("dtype", [np.int8, np.uint16, np.int32, np.uint32, np.uint64, np.float64, np.bool_],
                         ids=lambda d: np.dtype(d).name)
def test_every_kind_and_width(dtype):
    rng = np.random.default_rng(11)
    n = 70_001
    k = rng.integers(0, 70_000, n).astype(np.int32)  # a few rows a group: products stay small
    k[: n // 2] %= 40
    if np.dtype(dtype).kind == "f":
        v = rng.choice([-1.0, 1.0, 0.5, 2.0], n)
    else:
        v = rng.integers(0, 2, n).astype(dtype)
    T.assert_parity([HostCol(k % 700)], [(HostCol(v, rng.random(n) >= 0.2), ALL)], strategy=Strategy.PRIVATIZED)


@pytest.mark.parametrize("policy", [NullPolicy.EXCLUDE, NullPolicy.INCLUDE], ids=lambda p: p.name)
def test_two_word_keys_and_dictionary_values(policy):
    rng = np.random.default_rng(12)
    n = 100_003
    k1 = rng.integers(0, 9, n).astype(np.int64) * (1 << 40) - 1
    k2 = rng.choice([0.0, -0.0, np.nan, 1.5], n)
    keys = [HostCol(k1, rng.random(n) >= 0.1), HostCol(k2)]
    d = HostCol(rng.integers(0, 5, n).astype(np.int32), rng.random(n) >= 0.1,
                dict_keys=HostCol(np.array([-3, 8, 0, 77, 1 << 40], dtype=np.int64)))
    T.assert_parity(keys, [(d, SIX), (HostCol(rng.integers(0, 200, n).astype(np.uint8)), SIX)], policy,
                    Strategy.PRIVATIZED)


@pytest.mark.parametrize("rows,groups", [(100_000, 1500), (4_200_000, 700), (17_000_000, 1250), (17_000_000, 1990)])
def test_both_sides_of_the_line_to_atomics_a_row(rows, groups):
    """Tables above 1,024 slots: few accumulators go by rows (gbx_abi.cpp, tiled_pays)."""
    rng = np.random.default_rng(rows + groups)
    k = HostCol(rng.integers(0, groups, rows).astype(np.int64))
    v = HostCol(rng.integers(-100, 100, rows).astype(np.int64))
    w = HostCol(rng.integers(0, 50, rows).astype(np.float64), rng.random(rows) >= 0.1)
    for reqs in ([(v, [(Kind.COUNT_ALL, 0)])], [(v, [(Kind.SUM, 0)])], [(w, [(Kind.SUM, 0)])],
                 [(w, [(Kind.MIN, 0), (Kind.MAX, 0)])], [(v, [(Kind.SUM, 0), (Kind.MIN, 0), (Kind.MAX, 0)])]):
        T.assert_parity([k], reqs)


@pytest.mark.parametrize("rows,groups,hot", [(4_200_000, 300, 0.0), (4_200_000, 300, 0.3), (4_200_000, 3_000, 0.0),
                                             (4_200_000, 12_000, 0.015), (4_200_000, 12_000, 0.1), (4_200_000, 40_000, 0.1)])
def test_wide_plans_and_a_hot_key(rows, groups, hot):
    """Plans too wide for two tables an SM: bucketed, one run an SM, the global table, or the skewed form."""
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, rows).astype(np.int64)
    k[rng.random(rows) < hot] = groups // 2
    vals = [HostCol(rng.integers(-99, 99, rows).astype(np.float64), rng.random(rows) >= 0.1) for _ in range(5)]
    for aggs, cols in (([(Kind.SUM, 0), (Kind.COUNT_VALID, 0), (Kind.MEAN, 0)], vals),
                       ([(Kind.SUM, 0), (Kind.MIN, 0), (Kind.MAX, 0), (Kind.VARIANCE, 1)], vals[:3])):
        got, _ = T.assert_parity([HostCol(k)], [(v, aggs) for v in cols])
        assert got["stats"]["retries"] == 0
