"""Drop-in calls on pageable memory large enough for the threaded copy (24 MB
per copy): every byte arrives, whole or in slices, at sizes around the
threshold and around the copy's 1 MB chunks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nS,slices", [(3145727, 1), (3145728, 1), (3145729, 1), (4194305, 1), (13000001, 3)])
def test_threaded_host_copy(tbg, oracle, cuda, nS, slices):
    rng = np.random.default_rng(nS)
    n = 3300003  # R's copy is threaded too
    R = np.zeros(n, dtype=oracle.ROW)
    S = np.zeros(nS, dtype=oracle.ROW)
    R["key"] = rng.permutation(n)
    S["key"] = rng.integers(0, 2 * n, nS)
    want = int((S["key"] < n).sum())
    prev = tbg.set_dropin_slices(slices)
    try:
        assert tbg.find("RHO").join(R, S) == want
        S["key"][-1] ^= 1 << 31  # the last row counts: toggling its key moves the count by one
        want += 1 if S["key"][-1] < n else -1 if (S["key"][-1] ^ (1 << 31)) < n else 0
        assert tbg.find("PSM").join(R, S) == want
    finally:
        tbg.set_dropin_slices(prev)
    h2d, _ = tbg.last_transfer_bytes()
    assert h2d == 8 * (n + nS)
