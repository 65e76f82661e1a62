"""R relations that are not direct (direct.cu) because of keys that repeat side
by side or in one place: found before they queue at one word of the table."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join

pytestmark = pytest.mark.gpu


# two rows of one key side by side: in a 16-byte pair, across pairs, lanes,
# warps, rounds of 8192 rows, chunks, and at both ends; then far apart
@pytest.mark.parametrize("i,j", [(0, 1), (1, 2), (2, 3), (62, 63), (63, 64), (64, 65), (2047, 2048), (8191, 8192),
                                 (8192, 8193), (16383, 16384), (40010, 40011), (40011, 40012), (0, 40012), (777, 30000)])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("materialize", [False, True])
def test_one_repeated_key(tbg, oracle, cuda, i, j, off, materialize):
    rng = np.random.default_rng(i + j)
    R = np.zeros(40013, dtype=oracle.ROW)
    S = np.zeros(50021, dtype=oracle.ROW)
    R["key"] = 1000 + rng.permutation(len(R))
    R["key"][j] = R["key"][i]
    S["key"] = R["key"][rng.integers(0, len(R), len(S))]
    S["key"][:5] = R["key"][i]
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    m, _, st = run_join(tbg, cuda, "RHO", R, S, materialize=materialize, offset=off, cap=2 * len(S))
    assert m == oracle.rho(R, S)
    assert st.path == tbg.PATH_PARTITIONED


@pytest.mark.parametrize("algo", ["RHO", "RSM", "PSM"])
def test_hot_stretch_takes_no_longer(tbg, cuda, algo):
    """A quarter of R on one key, in one stretch: within one and a half times the
    join of rows that all come twice and 0.2 ms (with every row of the stretch
    entered it takes 0.6 ms more)."""
    torch = cuda
    nR, nS = 1 << 22, 1 << 23
    g = torch.Generator("cuda").manual_seed(1)
    cfg, st = tbg.config(algo), torch.cuda.current_stream().cuda_stream
    rows = lambda k: k | (torch.arange(len(k), device="cuda") << 32)  # noqa: E731
    S = torch.randint(0, nR, (nS,), device="cuda", generator=g)
    S[S == 5] = 6
    S = rows(S)

    def ms(k):
        R, best = rows(k), 1e9
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            tbg.join_device(cfg, R.data_ptr(), nR, S.data_ptr(), nS, stream=st)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    twice = (torch.arange(nR, device="cuda") // 2)[torch.randperm(nR, device="cuda", generator=g)]
    hot = torch.arange(nR, device="cuda")
    hot[-(nR // 4):] = 5
    assert ms(hot) <= 1.5 * ms(twice) + 0.2
