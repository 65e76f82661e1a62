"""Count-only RSM and PSM merge S with R's rows counted per key value.  The
sort-merge plans are selected with skew_split=0 (PSM) and fixed passes (RSM);
counts are whole numbers, equal to the oracle's."""
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


# digits that R's keys span in a partition: one key, the last span that the
# counters (19972 words) hold, the first that takes the sort, a wide one
@pytest.mark.parametrize("digits", [1, 2, 4096, 19972, 19973, 1 << 20])
@pytest.mark.parametrize("off", [0, 1])
def test_rsm_counter_spans(tbg, oracle, cuda, digits, off):
    rng = np.random.default_rng(digits)
    lo = 4294967295 - 2 * digits  # the top of the key range: key - smallest key must not wrap
    k = lo + 2 * rng.integers(0, digits, 3001)
    k[0], k[1] = lo, lo + 2 * (digits - 1)  # radix_bits = 1: one partition's digits are key >> 1
    R = rel(oracle, np.concatenate([k, k[:500]]), 0)  # duplicates
    S = rel(oracle, np.concatenate([lo - 40 + rng.integers(0, 2 * digits + 80, 50003), k, rng.integers(0, 100, 777)]), 1)
    m, _, _ = run_join(tbg, cuda, "RSM", R, S, offset=off, radix_bits=1, passes=1)
    assert m == oracle.rho(R, S)


# span of R's keys in bits (13: one radix bit; 21 and 28: two passes, 12 and 13
# low bits), R's smallest key (0, odd, the top of the range)
@pytest.mark.parametrize("bits", [13, 20, 21, 22, 28])
@pytest.mark.parametrize("base", ["zero", "odd", "top"])
def test_psm_bucket_counters(tbg, oracle, cuda, bits, base):
    rng = np.random.default_rng(bits)
    width = 1 << bits
    lo = {"zero": 0, "odd": 12345, "top": (1 << 32) - width}[base]
    k = lo + rng.integers(0, width, 60011)
    k[0], k[1] = lo, lo + width - 1
    R = rel(oracle, np.concatenate([k, k[:9000], np.full(3000, k[5])]), 0)  # duplicates and a heavy key
    pick = k[rng.integers(0, len(k), 200003)]
    other = rng.integers(0, 1 << 32, 50021)  # mostly outside R's range: they share buckets with R's keys
    S = rel(oracle, np.concatenate([pick, other, np.full(150001, k[6])]), 1)
    m, _, st = run_join(tbg, cuda, "PSM", R, S, skew_split=0)
    assert m == oracle.rho(R, S)
    assert st.passes == (3 if bits > 20 else 2)
