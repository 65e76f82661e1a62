"""The direct counting join (one bit per key value, S joined while it is read
for its histogram): RHO and RHT under the automatic plan, against the oracle
and against the partitioned join that a fixed number of passes selects.
Counts and partition statistics are whole numbers, so equality is exact."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import run_join, to_dev

pytestmark = pytest.mark.gpu


def relations(oracle, rng, nR, nS, lo, step, miss):
    """R: nR distinct keys lo + step * i in random order; S: a share `miss` of
    its rows has a key that R lacks (around and between R's keys)."""
    R = np.zeros(nR, dtype=oracle.ROW)
    S = np.zeros(nS, dtype=oracle.ROW)
    keys = (lo + step * np.arange(nR, dtype=np.uint64)) & 0xFFFFFFFF
    R["key"] = rng.permutation(keys)
    S["key"] = R["key"][rng.integers(0, nR, nS)]
    other = (lo - 50 + rng.integers(0, step * nR + 100, nS).astype(np.int64)) % (1 << 32)
    S["key"] = np.where(rng.random(nS) < miss, other, S["key"])
    oracle.fill_payloads(R, 0)
    oracle.fill_payloads(S, 1)
    return R, S


# |R|, |S|, smallest key, key step, misaligned: one row, sizes around a round of
# a CTA (8192 rows) and around the table's words, the table in shared memory
# (|R| up to 1.6 M) and in L2, ranges that start and end at the ends of 32 bits,
# sparse ranges that just fit (step 24) and that do not (step 40)
CASES = [(1, 1, 5, 1, 0), (1, 70000, 0, 1, 1), (31, 4097, 1, 1, 0), (33, 4095, 4294967295 - 32, 1, 1),
         (8191, 16385, 1, 1, 0), (8193, 65537, 31, 3, 1), (100003, 300007, 0, 24, 0), (100003, 300007, 1, 40, 1),
         (262144, 1 << 20, 1, 1, 0), (1500001, 3000017, 77, 1, 1), (3000001, 5000011, 1 << 31, 2, 0)]


@pytest.mark.parametrize("algo", ["RHO", "RHT"])
@pytest.mark.parametrize("nR,nS,lo,step,off", CASES)
def test_direct_join(tbg, oracle, cuda, algo, nR, nS, lo, step, off):
    rng = np.random.default_rng(nR + step)
    R, S = relations(oracle, rng, nR, nS, lo, step, 0.3)
    ref = oracle.rho(R, S)
    m, _, st = run_join(tbg, cuda, algo, R, S, offset=off)
    assert m == ref
    m2, _, st2 = run_join(tbg, cuda, algo, R, S, offset=off, passes=st.passes)  # the partitioned join
    assert m2 == ref
    for f in ("partitions", "work_items", "max_part_R", "max_part_S", "mean_part_R", "mean_part_S", "imbalance",
              "radix_bits", "passes"):
        assert getattr(st, f) == getattr(st2, f), f


@pytest.mark.parametrize("where", ["first", "last", "many", "all"])
def test_duplicate_keys_of_R_take_the_passes(tbg, oracle, cuda, where):
    """One duplicate that the careful first rounds see, one that only the
    count of set bits shows, many, and a relation of one key."""
    rng = np.random.default_rng(3)
    R, S = relations(oracle, rng, 400009, 700001, 1, 1, 0.2)
    if where == "first":
        R["key"][1] = R["key"][0]
    elif where == "last":
        R["key"][-1] = R["key"][-2]
    elif where == "many":
        R["key"] = rng.integers(1, 150000, len(R))
    else:
        R["key"], S = 9, S[:2000].copy()
        S["key"][::7] = 9
    ref = oracle.rho(R, S)
    m, _, st = run_join(tbg, cuda, "RHO", R, S)
    assert m == ref


def test_direct_outlier_outside_the_sample(tbg, oracle, cuda):
    """A key far outside the sampled range: not direct, same count."""
    rng = np.random.default_rng(4)
    R, S = relations(oracle, rng, 300000, 500000, 1, 1, 0.1)
    R["key"][7], S["key"][11] = 4000000000, 4000000000
    ref = oracle.rho(R, S)
    m, _, st = run_join(tbg, cuda, "RHO", R, S)
    assert m == ref


def test_direct_async_and_sliced(tbg, oracle, cuda):
    """Nothing waits in the asynchronous call and between the slices of the
    drop-in call: the passes are launched and step aside (or not)."""
    rng = np.random.default_rng(5)
    R, S = relations(oracle, rng, 60013, 250007, 1, 1, 0.25)
    D = R.copy()
    D["key"][0] = D["key"][1]
    s = cuda.cuda.current_stream().cuda_stream
    out = cuda.zeros(2, dtype=cuda.int64, device="cuda")
    tS, pS = to_dev(cuda, S)
    for k, rel in enumerate((R, D)):
        tR, pR = to_dev(cuda, rel)
        tbg.join_device_async(tbg.config("RHO"), pR, len(rel), pS, len(S), out.data_ptr() + 8 * k, stream=s)
        assert tbg.lib().tbg_sync_status(s) == 0
    refs = [oracle.rho(R, S), oracle.rho(D, S)]
    assert out.tolist() == refs
    prev = tbg.set_dropin_slices(5)
    try:
        assert [tbg.find("RHT").join(rel, S) for rel in (R, D)] == refs
    finally:
        tbg.set_dropin_slices(prev)


# ---------------------------------------------------------------- materialising
@pytest.mark.parametrize("algo", ["RHO", "RHT", "RSM", "PSM"])
@pytest.mark.parametrize("nR,nS,lo,step,off", [(1, 1, 5, 1, 0), (3, 70001, 0, 1, 1), (4095, 4097, 1, 1, 0),
                                               (8193, 65537, 31, 3, 1), (100003, 300007, 4294967295 - 1200036, 12, 1),
                                               (100003, 300007, 1, 40, 0), (1500001, 3000017, 77, 1, 1)])
def test_direct_rows(tbg, oracle, cuda, algo, nR, nS, lo, step, off):
    rng = np.random.default_rng(nR + step)
    R, S = relations(oracle, rng, nR, nS, lo, step, 0.3)
    ref, ref_rows = oracle.rho(R, S, materialize=True)
    m, rows, _ = run_join(tbg, cuda, algo, R, S, materialize=True, offset=off, cap=max(ref, 1))
    assert m == ref
    assert np.array_equal(oracle.sort_rows(rows), oracle.sort_rows(ref_rows))


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("short", [0, 1, 4097])
def test_direct_rows_stay_inside_the_buffer(tbg, oracle, cuda, shift, short):
    """Output buffers at every 4-byte phase of a 16-byte word and capacities
    below the row count: exact count, no word outside the buffer written."""
    rng = np.random.default_rng(7)
    R, S = relations(oracle, rng, 5003, 30011, 9, 2, 0.4)
    ref, ref_rows = oracle.rho(R, S, materialize=True)
    cap = ref - short
    tR, pR = to_dev(cuda, R, 1)
    tS, pS = to_dev(cuda, S)
    out = cuda.full((3 * ref + 64,), -7, dtype=cuda.int32, device="cuda")
    rc, m, _ = tbg.join_device(tbg.config("RHO", materialize=1), pR, len(R), pS, len(S), out.data_ptr() + 4 * (16 + shift),
                               cap, check=False)
    assert m == ref and rc == (tbg.ERR_CAPACITY if short else tbg.OK)
    host = out.cpu().numpy()
    a = 16 + shift
    assert (host[:a] == -7).all() and (host[a + 3 * cap:] == -7).all()
    got = oracle.sort_rows(host[a:a + 3 * cap].view(np.uint32).reshape(-1, 3))
    if not short:
        assert np.array_equal(got, oracle.sort_rows(ref_rows))
    else:  # cap distinct rows of the result
        code = lambda r: (r[:, 0].astype(np.uint64) << np.uint64(32)) | r[:, 2]  # noqa: E731
        assert len(np.unique(code(got))) == cap and np.isin(code(got), code(ref_rows)).all()


@pytest.mark.parametrize("case", ["empty_mark", "duplicate", "outlier", "zipf"])
@pytest.mark.parametrize("algo", ["RHO", "RSM", "PSM"])
def test_direct_rows_fall_back(tbg, oracle, cuda, algo, case):
    """A payload equal to the table's empty mark, a duplicate key and a key
    outside the sampled range send the join to the partitioned plan; a skewed
    S does not."""
    rng = np.random.default_rng(8)
    R, S = relations(oracle, rng, 20011, 90001, 1000, 1, 0.2)
    if case == "empty_mark":
        R["payload"][77] = 0xFFFFFFFF
        S["key"][5] = R["key"][77]
    elif case == "duplicate":
        R["key"][-1] = R["key"][0]
    elif case == "outlier":
        R["key"][3], S["key"][4] = 3000000000, 3000000000
    else:
        S["key"] = 1000 + np.minimum(rng.zipf(1.3, len(S)), 20010)
    ref, ref_rows = oracle.rho(R, S, materialize=True)
    m, rows, _ = run_join(tbg, cuda, algo, R, S, materialize=True, cap=ref)
    assert m == ref
    assert np.array_equal(oracle.sort_rows(rows), oracle.sort_rows(ref_rows))


def test_direct_rows_sliced(tbg, oracle, cuda):
    rng = np.random.default_rng(9)
    R, S = relations(oracle, rng, 60013, 250007, 1, 1, 0.25)
    ref, ref_rows = oracle.rho(R, S, materialize=True)
    prev = tbg.set_dropin_slices(3)
    try:
        c, rows = tbg.find("RHO").join(R, S, 2, materialize=True)
    finally:
        tbg.set_dropin_slices(prev)
    assert c == ref and np.array_equal(oracle.sort_rows(rows), oracle.sort_rows(ref_rows))


@pytest.mark.parametrize("materialize", [0, 1])
@pytest.mark.parametrize("nR", [5000, 90001])
def test_async_join_in_a_captured_graph(tbg, oracle, cuda, nR, materialize):
    """The asynchronous call captured into a CUDA graph (after a first call that
    sizes the scratch) and replayed on changing contents: distinct keys, then
    duplicates."""
    torch = cuda
    rng = np.random.default_rng(nR)
    R, S = relations(oracle, rng, nR, 120007, 1, 1, 0.3)
    D = R.copy()
    D["key"][0] = D["key"][1]
    tR, pR = to_dev(torch, R)
    tS, pS = to_dev(torch, S)
    tD, _ = to_dev(torch, D)
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    cap = 2 * len(S)
    rows = torch.zeros(3 * cap, dtype=torch.int32, device="cuda")
    st = torch.cuda.Stream()

    def call():
        tbg.join_device_async(tbg.config("RHO", materialize=materialize), pR, len(R), pS, len(S), out.data_ptr(),
                              rows.data_ptr() if materialize else 0, cap if materialize else 0, stream=st.cuda_stream)

    call()
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        call()
    for rel, dev in ((R, tR.clone()), (D, tD), (R, tR.clone())):
        tR.copy_(dev)
        torch.cuda.synchronize()
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        ref, ref_rows = oracle.rho(rel, S, materialize=True)
        assert out.item() == ref
        if materialize:
            got = rows[: 3 * ref].cpu().numpy().view(np.uint32).reshape(-1, 3)
            assert np.array_equal(oracle.sort_rows(got), oracle.sort_rows(ref_rows))
    assert tbg.lib().tbg_sync_status(st.cuda_stream) == 0


# |R| around one and two parts of the table in shared memory (P = 2^7 .. 2^9
# bins beside 55,808 .. 56,192 words of bits) and into L2, with S below one CTA
# round, with edge rows, and skewed
@pytest.mark.parametrize("nR", [1780000, 1803000, 3560001, 3610001])
@pytest.mark.parametrize("nS,z", [(4097, 0), (1000003, 0), (1000003, 1.2)])
def test_direct_table_parts(tbg, oracle, cuda, nR, nS, z):
    rng = np.random.default_rng(nR)
    R, S = relations(oracle, rng, nR, nS, 12345, 1, 0.2)
    if z:
        S["key"] = 12345 + np.minimum(rng.zipf(z, nS), nR + 5)
    want = int(((S["key"].astype(np.int64) >= 12345) & (S["key"].astype(np.int64) < 12345 + nR)).sum())
    for off in (0, 1):
        m, _, st = run_join(tbg, cuda, "RHO", R, S, offset=off)
        assert m == want
    _, _, st2 = run_join(tbg, cuda, "RHO", R, S, passes=st.passes)
    assert (st.max_part_R, st.max_part_S, st.work_items) == (st2.max_part_R, st2.max_part_S, st2.work_items)
