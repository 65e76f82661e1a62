"""Chained joins on device-resident output (the reference's three-way chain,
Enclave/TrustedJoins/secure_joins.cpp:348-399): R x S materialised,
to_relation of its rows as (key, R payload) tuples, then T x that relation.
Checked against the oracle's RHO run twice on the host."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gen_relation
from gpu_util import dev_to_host_rows, out_rows, rows_to_host, run_join, to_dev

pytestmark = pytest.mark.gpu


def _oracle_chain(oracle, R, S, T):
    c1, rows1 = oracle.rho(R, S, materialize=True)
    rel = np.zeros(c1, dtype=oracle.ROW)
    rel["key"] = rows1[:, 0]
    rel["payload"] = rows1[:, 1]
    c2, rows2 = oracle.rho(T, rel, materialize=True) if c1 and len(T) else (0, np.zeros((0, 3), np.uint32))
    return c1, rel, c2, rows2


def test_rows_to_relation(tbg, oracle, cuda):
    torch = cuda
    R = gen_relation(oracle, ("pk", 5000, 0, 0.0), 3, 0)
    S = gen_relation(oracle, ("fk", 20000, 5000, 0.0), 4, 1)
    c1, rel, _, _ = _oracle_chain(oracle, R, S, R[:0])
    m, rows, _ = run_join(tbg, torch, "RHO", R, S, materialize=True)
    assert m == c1
    # the GPU's rows back on the device, converted there
    flat = torch.from_numpy(np.ascontiguousarray(rows).reshape(-1).view(np.int32)).cuda()
    out = torch.zeros(max(m, 1), dtype=torch.int64, device="cuda")
    tbg.rows_to_relation(flat.data_ptr(), m, out.data_ptr())
    torch.cuda.synchronize()
    got = dev_to_host_rows(out, m)
    assert np.array_equal(got["key"], rows[:, 0]) and np.array_equal(got["payload"], rows[:, 1])


@pytest.mark.parametrize("kind", ["fk", "dup"])
def test_three_way_chain_matches_oracle(tbg, oracle, cuda, kind):
    torch = cuda
    rng = np.random.default_rng(7)
    R = gen_relation(oracle, ("pk", 1 << 16, 0, 0.0), 21, 0)
    S = gen_relation(oracle, ("fk", 1 << 18, 1 << 16, 0.0), 22, 1)
    if kind == "fk":
        T = gen_relation(oracle, ("pk", 1 << 16, 0, 0.0), 23, 0)
    else:  # T with duplicate keys: the second join multiplies rows
        T = np.zeros(50000, dtype=oracle.ROW)
        T["key"] = rng.integers(1, 30000, len(T))
        oracle.fill_payloads(T, 0)
    c1, _, c2, rows2 = _oracle_chain(oracle, R, S, T)
    tR, pR = to_dev(torch, R, 1)
    tS, pS = to_dev(torch, S)
    tT, pT = to_dev(torch, T)
    cap = c2 + 16
    tO, pO = out_rows(torch, cap)
    for algo in ("RHO", "LRN", "RSM"):
        m1, m2 = tbg.join_three_way(tbg.config(algo), pR, len(R), pS, len(S), pT, len(T), pO, cap,
                                    torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (m1, m2) == (c1, c2), algo
        got = rows_to_host(tO, m2)
        assert np.array_equal(oracle.sort_rows(got), oracle.sort_rows(rows2)), algo
    # count only
    m1, m2 = tbg.join_three_way(tbg.config("RHO"), pR, len(R), pS, len(S), pT, len(T))
    assert (m1, m2) == (c1, c2)


@pytest.mark.parametrize("nR,nS,nT,step", [(16385, 4095, 7, 1), (16387, 4097, 20000, 3), (20011, 300007, 17001, 1),
                                           (16385, 70001, 30000, 40)])
def test_three_way_chain_from_a_direct_join(tbg, oracle, cuda, nR, nS, nT, step):
    """The first join writes the relation itself when it is direct: output
    tiles that end unevenly, S rows without a partner, and (step 40) a key
    range too wide for it, whose rows are converted."""
    torch = cuda
    rng = np.random.default_rng(nR + nS)
    R, S, T = (np.zeros(n, dtype=oracle.ROW) for n in (nR, nS, nT))
    R["key"] = rng.permutation(100 + step * np.arange(nR))
    S["key"] = np.where(rng.random(nS) < 0.3, rng.integers(0, step * nR + 200, nS), R["key"][rng.integers(0, nR, nS)])
    T["key"] = rng.integers(0, step * nR + 200, nT)
    for rel, kind in ((R, 0), (S, 1), (T, 0)):
        oracle.fill_payloads(rel, kind)
    c1, _, c2, rows2 = _oracle_chain(oracle, R, S, T)
    tR, pR = to_dev(torch, R, 1)
    tS, pS = to_dev(torch, S)
    tT, pT = to_dev(torch, T)
    tO, pO = out_rows(torch, c2 + 16)
    for algo in ("RHO", "RHT", "PSM"):
        m1, m2 = tbg.join_three_way(tbg.config(algo), pR, nR, pS, nS, pT, nT, pO, c2 + 16,
                                    torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (m1, m2) == (c1, c2), algo
        assert np.array_equal(oracle.sort_rows(rows_to_host(tO, m2)), oracle.sort_rows(rows2)), algo


@pytest.mark.parametrize("nR", [1 << 20, 5000])
def test_chain_near_the_memory_limit(tbg, oracle, cuda, nR):
    """A selective chain whose first join's rows and passes fit, but not with
    room for |S| tuples beside them (which only a direct join could use)."""
    torch = cuda
    nS, nT = 1 << 25, 3001
    st = torch.cuda.Stream()
    S = torch.arange(nS, device="cuda") + (1 << 21) | (torch.arange(nS, device="cuda") << 32)
    S[-2000:] = torch.arange(2000, device="cuda") * 2 + 1
    R = torch.randperm(nR, device="cuda") | (torch.arange(nR, device="cuda") << 32)
    T = torch.arange(nT, device="cuda") | (torch.arange(nT, device="cuda") << 32)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # 12 B a row, two copies of S for the passes, R's, histograms and T x the
    # relation; each buffer with an eighth more where there is room, and no
    # room for the 8 B a row of |S| tuples (256 MB)
    need = nS * (12 + 16) + (96 << 20)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - need - need // 8, dtype=torch.uint8, device="cuda")
    try:
        got = tbg.join_three_way(tbg.config("RHO"), R.data_ptr(), nR, S.data_ptr(), nS, T.data_ptr(), nT, stream=st.cuda_stream)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert tuple(got) == (2000, 1500)  # T holds the odd keys up to 2999
