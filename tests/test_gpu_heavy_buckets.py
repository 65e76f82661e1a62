"""Count-only PSM on R relations whose rows crowd into few buckets (a hot key,
few distinct keys): their R rows are counted once.  Whole numbers: exact."""
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
    """The equi-join's rows (numpy: the oracle walks every row of a hot key's
    chain for every match)."""
    k, n = np.unique(R["key"], return_counts=True)
    at = np.minimum(np.searchsorted(k, S["key"]), len(k) - 1)
    return int(n[at][k[at] == S["key"]].sum())


# rows of one key around the line (32768 R rows), in the first, an inner and
# the last bucket, among spread keys (span in bits: one pass, two, 13 low bits)
@pytest.mark.parametrize("hot", [32700, 32768, 32769, 300001])
@pytest.mark.parametrize("bits,at", [(14, 0.0), (20, 0.5), (22, 1.0), (28, 0.3)])
def test_hot_key(tbg, oracle, cuda, hot, bits, at):
    rng = np.random.default_rng(hot + bits)
    lo, width = 977, 1 << bits
    key = lo + int(at * (width - 1))
    k = lo + rng.integers(0, width, 50021)
    k[0], k[1] = lo, lo + width - 1
    R = rel(oracle, rng.permutation(np.concatenate([k, np.full(hot, key)])), 0)
    S = rel(oracle, rng.permutation(np.concatenate([k[rng.integers(0, len(k), 90001)], np.full(200003, key),
                                                    rng.integers(0, 1 << 32, 30011)])), 1)
    for off in (0, 1):
        m, _, _ = run_join(tbg, cuda, "PSM", R, S, offset=off)
        assert m == count(R, S)


# ranges without bits above the low ones: two buckets that hold all of R
@pytest.mark.parametrize("values", [1, 2, 4, 5, 300, 4096])
@pytest.mark.parametrize("lo", [0, 4294967295 - 4095])
def test_few_values(tbg, oracle, cuda, values, lo):
    rng = np.random.default_rng(values)
    R = rel(oracle, lo + rng.integers(0, values, 250007), 0)
    S = rel(oracle, np.concatenate([lo + rng.integers(-5, values + 5, 300011), rng.integers(0, 1 << 32, 999)]) % (1 << 32), 1)
    m, _, _ = run_join(tbg, cuda, "PSM", R, S)
    assert m == count(R, S)


def test_many_heavy_buckets(tbg, oracle, cuda):
    """Every bucket heavy (about 80,000 rows of 4096 key values), then a
    smaller join on the same scratch."""
    rng = np.random.default_rng(2)
    R = rel(oracle, rng.integers(0, 1 << 16, 1300021), 0)
    S = rel(oracle, rng.integers(0, (1 << 16) + 900, 700001), 1)
    for n in (len(R), 66001):
        m, _, _ = run_join(tbg, cuda, "PSM", R[:n].copy(), S)
        assert m == count(R[:n], S)


def test_few_values_take_no_longer(tbg, cuda):
    """R's rows of a bucket are not counted once per S slice: the join takes
    at most twice as long as one of the same sizes with spread keys (it takes
    as long; with repeated counting five times)."""
    torch = cuda
    nR, nS = 1 << 23, 1 << 25
    g = torch.Generator("cuda").manual_seed(1)
    cfg, st = tbg.config("PSM"), torch.cuda.current_stream().cuda_stream

    def ms(values):
        R, S = (torch.randint(0, values, (n,), device="cuda", generator=g) | (torch.arange(n, device="cuda") << 32)
                for n in (nR, nS))
        best = 1e9
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            tbg.join_device(cfg, R.data_ptr(), nR, S.data_ptr(), nS, stream=st)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert ms(3000) <= 2 * ms(nR // 3)
