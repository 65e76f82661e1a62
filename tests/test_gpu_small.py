"""Joins whose R fits one table (at most 16384 rows) in one launch: against the
oracle and against the partitioned join that fixed passes select, whose
statistics they report.  Whole numbers: exact."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join, to_dev

pytestmark = pytest.mark.gpu


def relations(oracle, rng, nR, nS, kind):
    R = np.zeros(nR, dtype=oracle.ROW)
    S = np.zeros(nS, dtype=oracle.ROW)
    if kind == "dense":
        R["key"] = 4294967295 - rng.permutation(nR)
    elif kind == "sparse":
        R["key"] = rng.choice(1 << 32, nR, replace=False) if nR < 5000 else np.unique(rng.integers(0, 1 << 32, nR + 99))[:nR]
        rng.shuffle(R["key"])
    elif kind == "dup":
        R["key"] = rng.integers(0, max(1, nR // 3), nR)
    else:
        R["key"] = 7
    S["key"] = np.where(rng.random(nS) < 0.6, R["key"][rng.integers(0, nR, nS)],
                        (R["key"][0].astype(np.int64) - 99 + rng.integers(0, 2 * nR + 200, nS)) % (1 << 32))
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    return R, S


# around the tables (4096, 8192, 16384 rows; 16385 is not small) and a CTA's slice (2048 rows of S)
SHAPES = [(1, 1), (2, 2049), (4096, 2047), (4097, 300007), (8192, 2048), (8193, 50001), (16384, 100003), (16385, 100003)]


@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM"])
@pytest.mark.parametrize("kind", ["dense", "sparse", "dup"])
@pytest.mark.parametrize("nR,nS", SHAPES)
def test_small_join_counts(tbg, oracle, cuda, algo, kind, nR, nS):
    rng = np.random.default_rng(nR + nS)
    R, S = relations(oracle, rng, nR, nS, kind)
    ref = oracle.rho(R, S)
    off = nS & 1
    for _ in range(2):  # the kernel leaves its counters at zero
        m, _, st = run_join(tbg, cuda, algo, R, S, offset=off)
        assert m == ref
    m2, _, st2 = run_join(tbg, cuda, algo, R, S, offset=off, passes=1)
    assert m2 == ref
    for f in ("partitions", "work_items", "max_part_R", "max_part_S", "imbalance", "radix_bits", "passes"):
        assert getattr(st, f) == getattr(st2, f), f


@pytest.mark.parametrize("algo", ["RHO", "RSM"])
@pytest.mark.parametrize("kind", ["dense", "sparse", "dup", "one_key"])
@pytest.mark.parametrize("nR,nS", [(1, 1), (33, 2049), (4097, 9001), (16384, 30011)])
def test_small_join_rows(tbg, oracle, cuda, algo, kind, nR, nS):
    rng = np.random.default_rng(nR)
    if kind == "one_key":
        nR, nS = min(nR, 50), min(nS, 3001)
    R, S = relations(oracle, rng, nR, nS, kind)
    ref, ref_rows = oracle.rho(R, S, materialize=True)
    m, rows, st = run_join(tbg, cuda, algo, R, S, materialize=True, offset=1, cap=max(ref, 1))
    assert m == ref
    assert np.array_equal(oracle.sort_rows(rows), oracle.sort_rows(ref_rows))
    _, _, st2 = run_join(tbg, cuda, algo, R, S, materialize=True, offset=1, cap=max(ref, 1), passes=1)
    for f in ("partitions", "work_items", "max_part_R", "max_part_S"):
        assert getattr(st, f) == getattr(st2, f), f


def test_small_join_capacity_and_async(tbg, oracle, cuda):
    rng = np.random.default_rng(1)
    R, S = relations(oracle, rng, 5000, 40001, "dup")
    ref = oracle.rho(R, S)
    tR, pR = to_dev(cuda, R)
    tS, pS = to_dev(cuda, S)
    out = cuda.full((3 * ref,), -7, dtype=cuda.int32, device="cuda")
    rc, m, _ = tbg.join_device(tbg.config("RHO", materialize=1), pR, len(R), pS, len(S), out.data_ptr(), ref - 1000,
                               check=False)
    assert rc == tbg.ERR_CAPACITY and m == ref
    assert (out[3 * (ref - 1000):] == -7).all()
    counts = cuda.zeros(3, dtype=cuda.int64, device="cuda")
    s = cuda.cuda.current_stream().cuda_stream
    for k in range(3):
        tbg.join_device_async(tbg.config("RHO"), pR, len(R), pS, len(S), counts.data_ptr() + 8 * k, stream=s)
    assert tbg.lib().tbg_sync_status(s) == 0
    assert counts.tolist() == [ref] * 3
