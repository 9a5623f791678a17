"""The sorted kinds' row labels and NTH_ELEMENT's first / last rows
(gbx_sort.cu) against the oracle: label tables in shared memory and beyond it,
the all-ones key, two-word keys, excluded keys, and n = 0 / -1 under both null
policies beside another n."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from cudf_b200 import build
from cudf_b200._abi import Kind, NullPolicy
from oracle.oracle import HostCol
from tests import gbx_testing as T

pytestmark = pytest.mark.gpu


def _nth(n, policy):
    return (Kind.NTH_ELEMENT, n, {"null_policy": policy})


@pytest.mark.parametrize("n,groups", [(1, 1), (1023, 7), (70_001, 900), (1_100_000, 12_000), (1_100_003, 13_000)])
def test_labels_and_ends(n, groups):
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n).astype(np.int64) - 1  # -1: the all-ones word
    v = rng.integers(-1000, 1000, n).astype(np.int64)
    w = rng.standard_normal(n).astype(np.float32)
    aggs = [_nth(0, NullPolicy.INCLUDE), _nth(-1, NullPolicy.INCLUDE), _nth(0, NullPolicy.EXCLUDE),
            _nth(-1, NullPolicy.EXCLUDE), _nth(1, NullPolicy.EXCLUDE)]
    T.assert_parity([HostCol(k, rng.random(n) >= 0.05)],
                    [(HostCol(v), [(Kind.NUNIQUE, 0, {"null_policy": NullPolicy.EXCLUDE}), aggs[0], aggs[1]]),
                     (HostCol(w, rng.random(n) >= 0.4), aggs)])


def test_two_word_keys():
    rng = np.random.default_rng(3)
    n = 50_000
    keys = [HostCol(rng.integers(-2, 40, n).astype(np.int64)), HostCol(rng.integers(-1, 9, n).astype(np.int64))]
    T.assert_parity(keys, [(HostCol(rng.integers(0, 99, n).astype(np.int16)),
                            [_nth(0, NullPolicy.INCLUDE), _nth(-1, NullPolicy.EXCLUDE)])])


@pytest.mark.parametrize("n,groups", [(1600, 899), (1600, 900), (1600, 901), (70_000, 39_374),
                                      (70_000, 39_376), (5000, 5000)])
def test_few_rows_a_group(n, groups):
    """Both sides of the line between the label table and the global table (16 groups to 9 rows)."""
    rng = np.random.default_rng(n + groups)
    k = np.concatenate([np.arange(groups), rng.integers(0, groups, n - groups)])
    k = rng.permutation(k).astype(np.int64) * 31 - 31
    k[k == -31] = -1  # the all-ones word
    v = rng.integers(-1000, 1000, n).astype(np.int64)
    T.assert_parity([HostCol(k, rng.random(n) >= 0.01 if groups % 2 else None)],
                    [(HostCol(v), [(Kind.MEDIAN, 0), (Kind.NUNIQUE, 0, {"null_policy": NullPolicy.EXCLUDE}),
                                   _nth(0, NullPolicy.INCLUDE), _nth(1, NullPolicy.EXCLUDE)])])


def test_a_key_missing_from_the_table_is_reported():
    """sorted_kinds() on a hand-made table (tests/cpp/sorted_labels_test.cu)."""
    exe = build.LABELS_TEST_BIN
    if not os.path.exists(exe) or os.path.getmtime(exe) < max(map(os.path.getmtime, (build.LABELS_TEST_SRC, build.LIB))):
        build.build_labels_test()
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "0 failure(s)" in r.stdout, r.stdout + r.stderr
