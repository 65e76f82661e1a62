"""Which way a join went (tbg_stats.path and the batch's bit tables): the direct
and the one-launch joins report the statistics of the passes they do not take,
so only this field tells that they ran."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join, to_dev

pytestmark = pytest.mark.gpu


def relations(oracle, kind, nR=40013, nS=90001):
    rng = np.random.default_rng(21)
    step = {"step24": 24, "step64": 64}.get(kind, 1)
    lo = (1 << 32) - 7 * nR if kind == "top" else 1000
    R = np.zeros(nR, dtype=oracle.ROW)
    S = np.zeros(nS, dtype=oracle.ROW)
    R["key"] = lo + step * rng.permutation(nR).astype(np.int64)
    S["key"] = R["key"][np.minimum(rng.zipf(1.3, nS), nR) - 1] if kind == "zipf" else R["key"][rng.integers(0, nR, nS)]
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    if kind == "duplicate":
        R["key"][-1] = R["key"][0]
    elif kind == "outlier":
        R["key"][7] = 4000000000
    elif kind == "empty_mark":
        R["payload"][9] = 0xFFFFFFFF
    return R, S


DIRECT = {"dense", "step24", "top", "zipf", "empty_mark"}


@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM", "PSM", "LRN"])
@pytest.mark.parametrize("kind", sorted(DIRECT | {"step64", "duplicate", "outlier"}))
def test_path_counting(tbg, oracle, cuda, algo, kind):
    R, S = relations(oracle, kind)
    m, _, st = run_join(tbg, cuda, algo, R, S)
    assert m == oracle.rho(R, S)
    assert st.path == (tbg.PATH_DIRECT if kind in DIRECT else tbg.PATH_PARTITIONED)


@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM", "PSM"])
@pytest.mark.parametrize("kind", ["dense", "top", "zipf", "empty_mark", "step64", "duplicate", "outlier"])
def test_path_materialising(tbg, oracle, cuda, algo, kind):
    R, S = relations(oracle, kind)
    ref = oracle.rho(R, S)
    m, _, st = run_join(tbg, cuda, algo, R, S, materialize=True, cap=ref)
    assert m == ref
    direct = kind in DIRECT and kind != "empty_mark"  # a payload table cannot hold that payload
    assert st.path == (tbg.PATH_DIRECT if direct else tbg.PATH_PARTITIONED)


@pytest.mark.parametrize("cfg", [{"passes": 2}, {"radix_bits": 6}, {"skew_split": 0}])
@pytest.mark.parametrize("nR", [9000, 40013])
def test_path_of_fixed_plans(tbg, oracle, cuda, cfg, nR):
    R, S = relations(oracle, "dense", nR)
    m, _, st = run_join(tbg, cuda, "RHO", R, S, **cfg)
    assert m == len(S) and st.path == tbg.PATH_PARTITIONED


@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM"])
@pytest.mark.parametrize("materialize", [False, True])
@pytest.mark.parametrize("nR,small", [(1, True), (16384, True), (16385, False)])
def test_path_small(tbg, oracle, cuda, algo, materialize, nR, small):
    R, S = relations(oracle, "dense", nR)
    m, _, st = run_join(tbg, cuda, algo, R, S, materialize=materialize, cap=len(S))
    assert m == len(S)
    if algo == "RSM" and not materialize:  # one launch up to two partitions, of 2048 rows here
        small = nR <= 4096
    assert st.path == (tbg.PATH_SMALL if small else tbg.PATH_DIRECT)


def test_path_empty(tbg, oracle, cuda):
    R, S = relations(oracle, "dense")
    m, _, st = run_join(tbg, cuda, "RHO", R[:0], S)
    assert m == 0 and st.path == tbg.PATH_PARTITIONED


@pytest.mark.parametrize("kind,tables", [("dense", 3), ("duplicate", 0)])
def test_batch_reports_its_bit_tables(tbg, oracle, cuda, kind, tables):
    pairs = [relations(oracle, kind, n) for n in (77, 5000, 30011)]
    held = [(to_dev(cuda, R), to_dev(cuda, S)) for R, S in pairs]
    joins = [(r[1], len(R), s[1], len(S)) for (R, S), (r, s) in zip(pairs, held)]
    cuda.cuda.synchronize()
    b = tbg.Batch(joins, tbg.config("RHO", radix_bits=-1))
    try:
        assert b.describe()["bit_tables"] == tables
    finally:
        b.close()


def test_more_rows_than_key_values(tbg, oracle, cuda):
    """PSM knows R's range: more rows than key values are not tried (building
    their table took 8 of 79 us), as many distinct rows are."""
    launches = {}
    for nR, path in ((40000, tbg.PATH_DIRECT), (40001, tbg.PATH_PARTITIONED)):
        rng = np.random.default_rng(4)
        R = np.zeros(nR, dtype=oracle.ROW)
        S = np.zeros(60001, dtype=oracle.ROW)
        R["key"] = 77 + rng.permutation(nR) % 40000
        S["key"] = 77 + rng.integers(0, 40100, len(S))
        m, _, st = run_join(tbg, cuda, "PSM", R, S)
        assert m == oracle.rho(R, S) and st.path == path
        launches[nR] = st.kernel_launches
    # without the table's launches (clear, decide, one of two probes)
    assert launches[40001] == launches[40000] - 3
