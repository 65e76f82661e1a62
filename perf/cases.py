"""What is timed: equi-joins as users of the library run them, through the
Python package's public calls (tbg.join_device, tbg.join_three_way, tbg.Batch
and the drop-in tbg.find(name).join on host tables).

A case is a dict of plain values.  ``kind`` names the call:

  join   tbg.join_device, count only, with algorithm ``algo``
  rows   tbg.join_device, materialising, and the use the rows are made for:
         R's payload brought to S's row order (one column of |S| values)
  chain  tbg.join_three_way: R x S in device memory, its rows turned into a
         relation, T joined with it
  batch  tbg.Batch.run: many joins of uneven sizes planned once
  host   tbg.find(algo).join: the drop-in call on host (pageable) tables

The relations are those of the reference's generators (its pk, fk and Zipf
modes), made on the GPU from the seed: R is what a filter left of a table of
|R| * 100 / ``sel`` primary keys (or, with ``dup`` > 1, of a table that holds
every key dup times: a many-to-many join), S foreign keys of that table, or
Zipf-distributed over its keys with exponent ``z``.  With ``sparse`` the keys
are mapped by a bijection onto the whole 32-bit range, as hashed keys are.
"""
import importlib

import numpy as np
import torch

tbg = importlib.import_module("tee-bench_b200")


def _join(name, algo, nR, nS, sel=99, z=0.0, sparse=False, dup=1, kind="join"):
    c = {"kind": kind, "algo": algo, "nR": nR, "nS": nS, "sel": sel, "z": z, "sparse": sparse, "dup": dup}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: a lookup table against a micro-batch, where launches and latency count
        _join("rho_small", "RHO", 3000, 20011),
        # the equal-sized join of the benchmark (|R| = |S| = 2^21)
        _join("rho_c1", "RHO", 1 << 21, 1 << 21),
        # the headline join: 2^27 primary keys, 2^30 foreign keys
        _join("rho_c2", "RHO", 1 << 27, 1 << 30),
        # hashed keys over the whole 32-bit range, half of S without a partner, odd sizes
        _join("rho_sparse", "RHO", 16000057, 134217757, sel=50, sparse=True),
        # the histogram-table sibling on a dimension table of ordinary size, odd sizes
        _join("rht_odd", "RHT", 5000011, 100000037),
        # the sort-merge joins, large
        _join("rsm", "RSM", 1 << 25, 1 << 28),
        _join("psm", "PSM", 1 << 25, 1 << 28),
        # the learned join on the skewed workload it is made for (2^26 x 2^29, z = 1)
        _join("lrn_z1", "LRN", 1 << 26, 1 << 29, z=1.0),
        # materialised rows, used to bring a column of R to S's order
        _join("rows", "RHO", 3145735, 16777217, sel=80, kind="rows"),
        # a three-way chain on the device
        {"name": "chain", "kind": "chain", "algo": "RHO", "nR": 1 << 20, "nS": (1 << 24) + 3, "nT": 1500007, "sel": 99},
        # hundreds of joins of uneven sizes, replayed
        {"name": "batch", "kind": "batch", "njoins": 512, "lo": 10, "hi": 18, "zipf": 0.2},
        # the drop-in call on ordinary host memory, as a program of the reference makes it
        _join("host", "RHO", 1 << 22, 1 << 25, kind="host"),
    ]


def _log_uniform(rng, lo, hi):
    """An integer, odd or even, spread evenly over the logarithm of [2^lo, 2^hi]."""
    return int(round(2.0 ** rng.uniform(lo, hi)))


def draw(rng):
    kind = rng.choice(["join"] * 6 + ["rows", "chain", "batch", "host"])
    if kind == "batch":
        return {"kind": "batch", "njoins": _log_uniform(rng, 5, 9), "lo": 10, "hi": rng.choice([14, 16, 18]),
                "zipf": rng.choice([0.0, 0.2, 0.5])}
    sel = rng.choice([99, 99, 80, 50, 10])
    if kind == "chain":
        nR = _log_uniform(rng, 11, 20)
        return {"kind": "chain", "algo": rng.choice(["RHO", "RHT"]), "nR": nR,
                "nS": nR * rng.randint(1, 15) + rng.randint(0, 99), "nT": _log_uniform(rng, 11, 21), "sel": sel}
    if kind == "rows":
        nR = _log_uniform(rng, 12, 22)
        return _join(None, rng.choice(["RHO", "RHO", "RHT", "RSM", "PSM"]), nR, nR * rng.randint(1, 4) + rng.randint(0, 99),
                     sel, sparse=rng.random() < 0.25, kind="rows")
    if kind == "host":
        nR = _log_uniform(rng, 12, 22)
        return _join(None, rng.choice(["RHO", "RHT", "RSM", "PSM"]), nR, nR * rng.randint(1, 8) + rng.randint(0, 99), sel,
                     kind="host")
    algo = rng.choice(["RHO", "RHO", "RHO", "RHT", "RSM", "PSM", "LRN"])
    nR = _log_uniform(rng, 10, 26)
    nS = min(nR * rng.randint(1, 16) + rng.randint(0, 99), 1 << 29)
    z = rng.choice([0.0, 0.0, 0.5, 1.0, 1.5]) if algo != "LRN" else rng.choice([0.5, 1.0, 1.5])
    dup = rng.choice([1, 1, 1, 1, 1, 3]) if z == 0.0 else 1
    return _join(None, algo, nR, nS, 99 if z else sel, z, rng.random() < 0.25 and nR <= 1 << 24, dup)


# ---------------------------------------------------------------- inputs
def _stream():
    return torch.cuda.current_stream().cuda_stream


def _spread(t):
    """Maps the keys (low halves) of rows onto the 32-bit range by a bijection, in place."""
    for part in t.split(1 << 24):
        k = part & 0xFFFFFFFF
        part -= k
        k ^= k >> 16
        k = (k * 0x9E3779B1) & 0xFFFFFFFF
        k ^= k >> 15
        part += k
    return t


def _rows(n):
    return torch.empty(n, dtype=torch.int64, device="cuda")


def _relations(case, seed):
    nR, nS, dup = case["nR"], case["nS"], case.get("dup", 1)
    table = nR * 100 // case["sel"]
    keys = table // dup
    R, S, st = _rows(table), _rows(nS), _stream()
    if dup > 1:
        tbg.gen_fk(R.data_ptr(), table, keys, 2 * seed + 1, st)
        R = R[torch.randperm(table, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))[:nR]]
    else:
        tbg.gen_pk(R.data_ptr(), table, 2 * seed + 1, st)
        R = R[:nR]
    if case.get("z"):
        tbg.gen_zipf(S.data_ptr(), nS, keys, case["z"], 1, 2 * seed + 2, st)
    else:
        tbg.gen_fk(S.data_ptr(), nS, keys, 2 * seed + 2, st)
    if case.get("sparse"):
        _spread(R), _spread(S)
    return R, S


def _host(t):
    return t.cpu().numpy().view(tbg.ROW)


def _batch_joins(case, seed):
    rs = np.random.RandomState(seed % (1 << 32))
    n = case["njoins"]
    nR = np.round(2.0 ** rs.uniform(case["lo"], case["hi"], n)).astype(np.int64)
    nS = nR * rs.randint(1, 17, n)
    zipf = rs.random_sample(n) < case["zipf"]
    buf, st, at, joins = _rows(int(nR.sum() + nS.sum())), _stream(), 0, []
    for i in range(n):
        pR = buf.data_ptr() + 8 * at
        pS = pR + 8 * int(nR[i])
        at += int(nR[i] + nS[i])
        tbg.gen_pk(pR, int(nR[i]), 3 * (seed + 1000 * i) + 1, st)
        if zipf[i]:
            tbg.gen_zipf(pS, int(nS[i]), int(nR[i]), 1.0, 0, 3 * (seed + 1000 * i) + 2, st)
        else:
            tbg.gen_fk(pS, int(nS[i]), int(nR[i]), 3 * (seed + 1000 * i) + 2, st)
        joins.append((pR, int(nR[i]), pS, int(nS[i])))
    return buf, joins


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        buf, joins = _batch_joins(case, seed)
        return {"kind": kind, "buf": buf, "batch": tbg.Batch(joins, stream=_stream()),
                "counts": torch.zeros(len(joins), dtype=torch.int64, device="cuda")}
    R, S = _relations(case, seed)
    s = {"kind": kind, "R": R, "S": S, "nR": case["nR"], "nS": case["nS"]}
    if kind == "host":
        s.update(R=_host(R), S=_host(S), join=tbg.find(case["algo"]))
        return s
    s["cfg"] = tbg.config(case["algo"], materialize=int(kind == "rows"))
    if kind == "rows":
        s["out"] = torch.empty(3 * case["nS"], dtype=torch.int32, device="cuda")
        s["column"] = torch.full((case["nS"],), -1, dtype=torch.int32, device="cuda")
    if kind == "chain":
        s["T"], s["nT"] = _rows(case["nT"]), case["nT"]
        tbg.gen_pk(s["T"].data_ptr(), case["nT"], 2 * seed + 3, _stream())
    return s


def run(s):
    kind = s["kind"]
    if kind == "host":
        return s["join"].join(s["R"], s["S"])
    st = _stream()
    if kind == "batch":
        s["batch"].run(s["counts"].data_ptr(), st)
        return s["counts"]
    pR, pS = s["R"].data_ptr(), s["S"].data_ptr()
    if kind == "chain":
        return tbg.join_three_way(s["cfg"], pR, s["nR"], pS, s["nS"], s["T"].data_ptr(), s["nT"], stream=st)
    if kind == "rows":
        _, m, _ = tbg.join_device(s["cfg"], pR, s["nR"], pS, s["nS"], s["out"].data_ptr(), s["nS"], stream=st)
        rows = s["out"][: 3 * m].view(-1, 3)
        s["column"][rows[:, 2].long()] = rows[:, 1]  # S's payload is its row number
        return m, s["column"]
    return tbg.join_device(s["cfg"], pR, s["nR"], pS, s["nS"], stream=st)[1]


def work(case):
    """Every relation read once and the result written once."""
    kind = case["kind"]
    if kind == "batch":
        # |R| = 2^U, |S| = 8.5 |R| on average
        mean = (2.0 ** case["hi"] - 2.0 ** case["lo"]) / ((case["hi"] - case["lo"]) * np.log(2.0))
        return {"bytes": float(case["njoins"] * (mean * 9.5 * 8 + 8)), "flops": 0.0}
    rows = case["nR"] + case["nS"] + case.get("nT", 0)
    out = 8.0
    if kind == "rows":
        out = case["nS"] * (12 * case["sel"] / 100 + 4)
    return {"bytes": 8.0 * rows + out, "flops": 0.0}


# ---------------------------------------------------------------- reference values
def _keys(t):
    return (t & 0xFFFFFFFF).sort()


def _matches(R, S):
    """Rows of the equi-join of two relations (row tensors), in 64 bits."""
    k = _keys(R)[0]
    q = S & 0xFFFFFFFF
    return int((torch.searchsorted(k, q, right=True) - torch.searchsorted(k, q)).sum())


def exact(case, seed):
    if case["kind"] == "batch":
        buf, joins = _batch_joins(case, seed)
        if case["njoins"] > 64:
            return None
        base = buf.data_ptr()
        part = lambda p, n: buf[(p - base) // 8:(p - base) // 8 + n]  # noqa: E731
        return torch.tensor([_matches(part(a, n), part(b, m)) for a, n, b, m in joins])
    if case["nR"] + case["nS"] > 1 << 26:
        return None
    R, S = _relations(case, seed)
    m = _matches(R, S)
    if case["kind"] == "chain":
        # T holds 1..nT once each: every row of R x S whose key is at most nT matches once
        return m, _matches(R, S[(S & 0xFFFFFFFF) <= case["nT"]])
    if case["kind"] == "rows":
        k, order = _keys(R)
        q = S & 0xFFFFFFFF
        at = torch.searchsorted(k, q).clamp(max=len(k) - 1)
        return m, torch.where(k[at] == q, R[order[at]] >> 32, -1).to(torch.int32)
    return m
