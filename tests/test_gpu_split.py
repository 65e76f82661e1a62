"""Keys that share their low bits fall into one partition, or a few, of the radix
join: its S side is split over the SMs for every chunk of its R side.  Whole
numbers and rows: exact."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join

pytestmark = pytest.mark.gpu


def relations(oracle, nR, nS, stride):
    rng = np.random.default_rng(nR + stride)
    R = np.zeros(nR, dtype=oracle.ROW)
    S = np.zeros(nS, dtype=oracle.ROW)
    R["key"] = rng.permutation(nR).astype(np.uint32) * np.uint32(stride)
    S["key"] = np.where(rng.random(nS) < 0.9, R["key"][rng.integers(0, nR, nS)], rng.integers(0, 1 << 32, nS))
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    return R, S


# R chunks of a partition: 1 (its table is never too small), a few, many; S
# rows a few and many per chunk; with fewer partitions than SMs and with more
@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM", "LRN"])
@pytest.mark.parametrize("materialize", [False, True])
@pytest.mark.parametrize("nR,nS,stride", [(20011, 70001, 1 << 16), (65536, 100003, 1 << 16), (65536, 262147, 1 << 12),
                                          (131073, 400009, 1 << 11), (40013, 3001, 1 << 15)])
def test_one_partition(tbg, oracle, cuda, algo, materialize, nR, nS, stride):
    R, S = relations(oracle, nR, nS, stride)
    if materialize:
        ref, ref_rows = oracle.rho(R, S, materialize=True)
        m, rows, st = run_join(tbg, cuda, algo, R, S, materialize=True, cap=ref)
        assert np.array_equal(oracle.sort_rows(rows), oracle.sort_rows(ref_rows))
    else:
        ref = oracle.rho(R, S)
        m, _, st = run_join(tbg, cuda, algo, R, S)
    assert m == ref and st.path == tbg.PATH_PARTITIONED


@pytest.mark.parametrize("algo", ["RHO", "RSM"])
@pytest.mark.parametrize("materialize", [False, True])
@pytest.mark.parametrize("nR,nS,stride", [(65536, 262144, 1 << 16), (131072, 524288, 1 << 12), (65536, 1048576, 1 << 13)])
def test_one_partition_fills_the_gpu(tbg, oracle, cuda, algo, materialize, nR, nS, stride):
    """The work items of the one partition that holds nearly all rows are more
    than half of a 148-SM GPU's CTAs at one per SM (its R chunks alone are 4 to
    32 items); at most half of S as finely split as one-chunk partitions."""
    R, S = relations(oracle, nR, nS, stride)
    m, _, st = run_join(tbg, cuda, algo, R, S, materialize=materialize, cap=nS)
    assert st.partitions < 148 and st.max_part_R > 0.9 * nR / max(1, 2 ** 13 // stride)
    assert st.work_items >= 74
