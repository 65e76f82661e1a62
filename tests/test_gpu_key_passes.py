"""Counting joins that partition bare keys, and the build/probe's table of
32-bit cells: RHO and RHT with a fixed number of passes, against the oracle.
Counts are whole numbers, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join

pytestmark = pytest.mark.gpu


def tables(oracle, seed, nR, nS, lo, hi):
    """Keys drawn with repetition from [lo, hi): duplicates on both sides."""
    rng = np.random.default_rng(seed)
    R, S = np.zeros(nR, dtype=oracle.ROW), np.zeros(nS, dtype=oracle.ROW)
    R["key"] = rng.integers(lo, hi, nR)
    S["key"] = rng.integers(lo, hi, nS)
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    return R, S


# rows around the tiles of the first pass (4096 rows) and of the second (8192
# keys), one row, ragged sizes, and enough keys for many units of odd starts
@pytest.mark.parametrize("passes,bits", [(1, 5), (2, 6), (2, 11), (2, 14)])
@pytest.mark.parametrize("nR,nS,off", [(1, 4095, 1), (4097, 8191, 0), (8193, 4096, 1), (20011, 70003, 0), (300007, 500009, 1)])
def test_key_passes(tbg, oracle, cuda, passes, bits, nR, nS, off):
    R, S = tables(oracle, nR + bits, nR, nS, 0, max(4, nR // 2))
    for algo in ("RHO", "RHT"):
        assert run_join(tbg, cuda, algo, R, S, offset=off, passes=passes, radix_bits=bits)[0] == oracle.rho(R, S), algo


# R partitions around the two table sizes (10240 and 16384 rows) and beyond
# them, on 32-bit keys, with keys that repeat and the extreme ones
@pytest.mark.parametrize("rows", [10239, 10240, 10241, 16383, 16384, 16385, 40000])
@pytest.mark.parametrize("spread", [1 << 32, 9000])
def test_cell_tables(tbg, oracle, cuda, rows, spread):
    R, S = tables(oracle, rows, 2 * rows, 50021, 0, spread)
    R["key"] = R["key"] & ~np.uint32(1) | (np.arange(2 * rows) & 1).astype(np.uint32)  # two partitions of `rows`
    S["key"][::3] = R["key"][np.arange(len(S["key"][::3])) % (2 * rows)]
    R["key"][:2] = S["key"][:2] = (0xFFFFFFFE, 0xFFFFFFFF)
    assert run_join(tbg, cuda, "RHO", R, S, radix_bits=1, passes=1)[0] == oracle.rho(R, S)
