"""The plans of the sort-merge joins that joins with small or distinct keys no
longer take: the merge of globally sorted relations with runs of equal keys
longer than its tiles, and the LSD passes of a bucket past a million rows.
Whole numbers and rows: exact, against numpy."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join

pytestmark = pytest.mark.gpu


def rel(oracle, keys, kind):
    t = np.zeros(len(keys), dtype=oracle.ROW)
    t["key"] = np.asarray(keys, dtype=np.uint64) & 0xFFFFFFFF
    oracle.fill_payloads(t, kind)
    return t


def count(R, S):
    k, n = np.unique(R["key"], return_counts=True)
    at = np.minimum(np.searchsorted(k, S["key"]), len(k) - 1)
    return int(n[at][k[at] == S["key"]].sum())


def rows_of(R, S):
    """The join's rows, sorted: every S row beside each R row of its key."""
    R, S = np.sort(R, order=["key", "payload"]), np.sort(S, order=["key", "payload"])
    a, b = np.searchsorted(R["key"], S["key"]), np.searchsorted(R["key"], S["key"], side="right")
    n = b - a
    s = np.repeat(np.arange(len(S)), n)
    r = np.repeat(a, n) + np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)
    return sort_rows(np.stack([R["key"][r], R["payload"][r], S["payload"][s]], axis=1))


def sort_rows(x):
    return x[np.lexsort((x[:, 2], x[:, 1], x[:, 0]))]


# rows of each key of R: around the four steps that are walked back, a tile and
# several tiles of the merge; the 32-bit range is past the MSD sort's 28 bits,
# so both relations are sorted by the LSD passes and merged
@pytest.mark.parametrize("run", [2, 4, 5, 6, 63, 1000, 4096, 30011])
@pytest.mark.parametrize("off", [0, 1])
def test_counting_merge_runs(tbg, oracle, cuda, run, off):
    rng = np.random.default_rng(run)
    keys = rng.choice(1 << 32, 1 + 300000 // run, replace=False)
    keys[0], keys[-1] = 3, (1 << 32) - 2
    r = np.concatenate([np.repeat(keys, run), rng.integers(0, 1 << 32, 5003)])
    s = np.concatenate([keys[rng.integers(0, len(keys), 200003)], np.repeat(keys[:9], 5000), rng.integers(0, 1 << 32, 999)])
    R, S = rel(oracle, rng.permutation(r), 0), rel(oracle, rng.permutation(s), 1)
    m, _, st = run_join(tbg, cuda, "PSM", R, S, offset=off)
    assert m == count(R, S)
    assert st.path == tbg.PATH_PARTITIONED and st.passes == 4 and st.partitions == 0  # LSD passes over 32 bits


# a bucket past 2^20 rows in R, in S, in both: a 28-bit range takes two passes
# and the bucket sort (three in all), the LSD passes of such a relation four
@pytest.mark.parametrize("where,hot_R,hot_S", [("R", 1 << 20, 3), ("R", (1 << 20) + 1, 3), ("S", 2, (1 << 20) + 1),
                                               ("both", (1 << 20) + 5, 1), ("none", 1000, 1000)])
def test_materialising_heavy_bucket_takes_lsd(tbg, oracle, cuda, where, hot_R, hot_S):
    rng = np.random.default_rng(hot_R)
    lo, width = 5, 1 << 28
    hot = lo + 12345678
    r = lo + rng.integers(0, width, 200003)
    r[0], r[1], r[2] = lo, lo + width - 1, r[3]  # R's range and a key that comes twice: not direct
    r = r[(r - lo) >> 13 != (hot - lo) >> 13]  # the hot key alone in its bucket
    s = r[rng.integers(0, len(r), 150001)]
    if where == "both":  # S's heavy bucket holds a key beside R's heavy one
        s = np.concatenate([s, np.full((1 << 20) + 1, hot + 1)])
    R = rel(oracle, rng.permutation(np.concatenate([r, np.full(hot_R, hot)])), 0)
    S = rel(oracle, rng.permutation(np.concatenate([s, np.full(hot_S, hot)])), 1)
    ref = count(R, S)
    m, rows, st = run_join(tbg, cuda, "PSM", R, S, materialize=True, cap=ref)
    assert m == ref and st.path == tbg.PATH_PARTITIONED
    assert np.array_equal(sort_rows(rows), rows_of(R, S))
    assert st.passes == (4 if max(hot_R, hot_S) > 1 << 20 else 3)
