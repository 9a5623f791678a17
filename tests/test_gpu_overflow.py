"""Groupbys whose sample misses most of the groups: the table overflows, the
pass is redone with a larger one, and the result is the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from cudf_b200._abi import Kind, Strategy
from oracle.oracle import HostCol
from tests import gbx_testing as T

pytestmark = pytest.mark.gpu

AGGS = [(Kind.SUM, 0), (Kind.COUNT_ALL, 0), (Kind.MAX, 0)]


def _keys(n, seen, dtype=np.int64):
    """n distinct keys but for the 65,536 sampled rows, which hold `seen` keys."""
    m = 1 << 16
    k = np.arange(n, dtype=dtype) + 1000
    at = ((np.arange(m) + 0.5) * n / m).astype(np.int64)
    k[at] = np.arange(m) % seen
    return k


@pytest.mark.parametrize("strategy", [None, Strategy.GLOBAL, Strategy.PRIVATIZED, Strategy.WARP, Strategy.BUCKETED],
                         ids=lambda s: "auto" if s is None else s.name)
@pytest.mark.parametrize("two_words", [False, True], ids=["one_word", "two_words"])
def test_overflowing_table(strategy, two_words):
    n = 300_000
    keys = [HostCol(_keys(n, 500))]
    if two_words:
        keys.append(HostCol(-3 * _keys(n, 500)))
    v = np.arange(n, dtype=np.int64) % 1000
    got, want = T.assert_parity(keys, [(HostCol(v), AGGS)], strategy=strategy)
    assert got["stats"]["retries"] >= 1
    assert got["num_groups"] == want["num_groups"]


def test_overflow_of_a_wide_skewed_plan():
    """Bucketed for the 300 keys the sample sees; the other 20,000 overflow its table, and the skewed form, which
    spills them to a larger global table, takes over."""
    n, m = 4_300_000, 1 << 16
    rng = np.random.default_rng(5)
    k = rng.integers(0, 20_000, n)
    k[((np.arange(m) + 0.5) * n / m).astype(np.int64)] = np.arange(m) % 300
    cols = [HostCol(rng.integers(-50, 50, n).astype(np.float64), rng.random(n) >= 0.1) for _ in range(3)]
    aggs = [(Kind.SUM, 0), (Kind.MIN, 0), (Kind.MAX, 0), (Kind.VARIANCE, 1)]
    got, _ = T.assert_parity([HostCol(k.astype(np.int64))], [(c, aggs) for c in cols])
    assert got["stats"]["retries"] == 1 and got["stats"]["strategy"] == Strategy.PRIVATIZED
