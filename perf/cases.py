"""The work that a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; its "kind" says which public call it makes:

  witness    auto.dp_witness(p, order)                 columns of a minimum logical
  distance   auto.dp_distance(p, order)                every observable's exact distance, planning included
  sweep      kernel.CompiledPlan execute + result      one scheduled sweep with a table kept at a checkpoint
  batch      batch.batched_dp_distances(problems)      many instances in one persistent launch
  tree       tree_dp.CompiledTreeDP.run(target)        least weight of several targets on one compiled tree
  sparse     sparse_dp.query(trellis, K)               meet in the middle at one threshold
  search     search.distance(p, k_table, kmax)         weight-bounded search with its completion table
  table      search.Table(p, k).lookup(...)            completion table built and probed

Every output is a whole number, so a value is either the same or wrong.
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from tropidist_gb300 import auto, batch, device, kernel, search, sparse_dp, synth, tree_dp
from tropidist_gb300.problem import Problem, dedupe

LIMITS = dict(max_join_work=None, max_memory_bytes=None, max_seconds=None)


def listed():
    return [
        # the CPU-runnable problem size (m=120, n=240, window 16, one logical row): the smallest whole
        # call, bound by launches and by one block's latency
        dict(name="witness_bits15", kind="witness", m=120, n=240, window=16, nobs=1, bits=15, weights=False),
        # an ordinary code with a dozen observables: narrow tables, many short launches, odd sizes
        dict(name="distance_bits19", kind="distance", m=161, n=333, window=22, nobs=12, bits=19, weights=False),
        # weighted columns (1, 2, 3) whose sum passes 254: 16-bit tables
        dict(name="distance_u16_bits24", kind="distance", m=300, n=601, window=28, nobs=4, bits=24, weights=True),
        # m=1000, n=2000, window 30: tables of 64 MB, which fit L2 one at a time
        dict(name="sweep_bits26", kind="sweep", m=1000, n=2000, window=30, bits=26, dtype="u8"),
        # 16-bit tables of 256 MB
        dict(name="sweep_u16_bits27", kind="sweep", m=500, n=999, window=31, bits=27, dtype="u16"),
        # the benchmark's shape (window 37): 2 GB tables, bound by HBM
        dict(name="sweep_bits31", kind="sweep", m=1000, n=2000, window=37, bits=31, dtype="u8"),
        # uneven instances (widths about 12-26, 1-12 observables each) submitted together
        dict(name="batch_48", kind="batch", count=48, wmin=12, wmax=26, max_obs=12),
        # tree DP of one compiled logical query, several targets on the same tree
        dict(name="tree_n240", kind="tree", m=120, n=240, window=16, targets=4, lo=2e9, hi=8e9),
        # circuit-style detector error models: states of one word, and of three words
        dict(name="sparse_s37_K6", kind="sparse", rounds=20, checks=24, ncols=5000, K=6),
        dict(name="sparse_s140_K5", kind="sparse", rounds=10, checks=150, ncols=4001, K=5),
        # rotated surface code, table of all triples
        dict(name="search_d13", kind="search", d=13, k=3),
        # completion table of all triples of 301 columns (4.5 M subsets) and a million probes
        dict(name="table_n301_k3", kind="table", m=120, n=301, window=40, k=3, probes=1000003),
    ]


def _between(rng, lo, hi):
    """A whole number, spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


# (window, peak bits) of the banded generator's natural order: the peak is 0.83-0.9 of the window
def _window(bits):
    return int(round(bits / 0.87))


def draw(rng):
    kind = rng.choice(["witness", "distance", "distance", "sweep", "sweep", "sweep", "batch", "tree", "sparse",
                       "search", "table"])
    if kind == "witness":
        bits, n = rng.randint(10, 16), _between(rng, 120, 600)
        return dict(kind=kind, m=n // 2, n=n, window=_window(bits), nobs=rng.randint(1, 3), bits=bits,
                    weights=rng.random() < 0.3)
    if kind == "distance":
        bits, n = rng.randint(12, 25), _between(rng, 160, 900)
        return dict(kind=kind, m=n // 2, n=n, window=_window(bits), nobs=rng.randint(3, 12), bits=bits,
                    weights=rng.random() < 0.4)
    if kind == "sweep":
        u16 = rng.random() < 0.35
        bits, n = rng.randint(17, 26 if u16 else 30), _between(rng, 400, 2000)
        return dict(kind=kind, m=n // 2, n=n, window=_window(bits), bits=bits, dtype="u16" if u16 else "u8")
    if kind == "batch":
        return dict(kind=kind, count=_between(rng, 6, 48), wmin=rng.randint(10, 14), wmax=rng.randint(18, 26),
                    max_obs=rng.randint(2, 12))
    if kind == "tree":
        n = rng.randint(90, 250)
        return dict(kind=kind, m=n // 2, n=n, window=rng.randint(8, 15), targets=rng.randint(1, 6), lo=0, hi=8e9)
    if kind == "sparse":
        wide = rng.random() < 0.5
        return dict(kind=kind, rounds=rng.randint(6, 20), checks=rng.randint(60, 150) if wide else rng.randint(12, 28),
                    ncols=_between(rng, 1000, 4000), K=rng.randint(3, 5 if wide else 6))
    if kind == "search":
        return dict(kind=kind, d=rng.choice([7, 9, 11, 13]), k=rng.choice([2, 3]))
    n = _between(rng, 80, 300)
    return dict(kind="table", m=n // 2, n=n, window=rng.randint(20, 40), k=rng.choice([2, 3]),
                probes=_between(rng, 10000, 1000000))


# ---------------------------------------------------------------------- inputs
def _weighted(p, seed):
    p.weights = [int(x) for x in np.random.default_rng([seed, 7]).integers(1, 4, p.ncols)]
    return p


def _banded(case, seed, nobs):
    """The first of the seed's banded problems whose sweeps peak at case["bits"] bits, the order and
    the plans; the nearest of 40 where none does."""
    best = None
    for k in range(40):
        p = synth.banded(case["m"], case["n"], case["window"], 3, nobs, seed=1000 * seed + k)
        order = list(range(p.ncols))
        plans = [pl for _, pl in auto._plans(p, order)]
        off = abs(max([pl.peak_bits for pl in plans if pl.feasible] or [-99]) - case["bits"])
        if best is None or off < best[0]:
            best = (off, p)
        if off == 0:
            break
    p = best[1]
    if case.get("weights") or case.get("dtype") == "u16":
        _weighted(p, seed)
    return p, order, [pl for _, pl in auto._plans(p, order)]


def _balanced(xs):
    if len(xs) == 1:
        return xs[0]
    m = len(xs) // 2
    return _balanced(xs[:m]), _balanced(xs[m:])


def _tree(case, seed):
    """A logical query on the balanced tree, the first of the seed's problems in the range of work, and
    targets: the logical query itself and syndromes of random column sets."""
    best = None
    for k in range(20):
        p = synth.banded(case["m"], case["n"], case["window"], 3, 1, seed=1000 * seed + k)
        cols, nrows = tree_dp._augmented(p.h, p.l, 1)
        prog = tree_dp.CompiledTreeDP(cols, _balanced(list(range(p.ncols))))
        work = prog.preflight(max_join_work=None, max_memory_bytes=None)["join_work"]
        off = max(case["lo"] - work, work - case["hi"], 0)
        if best is None or off < best[0]:
            best = (off, prog, work, nrows, p)
        if off == 0:
            break
    _, prog, work, nrows, p = best
    rng = np.random.default_rng([seed, 3])
    targets = [1 << nrows]
    while len(targets) < case["targets"]:
        t = 0
        for j in rng.choice(p.ncols, size=p.ncols // 2, replace=False):
            t ^= prog_column(p, nrows, int(j))
        targets.append(t)
    return prog, targets[:case["targets"]], work


def prog_column(p, nrows, j):
    return p.h[j] | ((p.l[j] & 1) << nrows)


def _surface(d, seed):
    """Rotated surface code of distance d: the checks of one type as rows in a random order, the logical
    row a column of qubits times random checks of the other type."""
    rng = np.random.default_rng([seed, 5])
    q = lambda r, c: r * d + c
    mine, other = [], []
    for r in range(d + 1):
        for c in range(d + 1):
            qs = [q(a, b) for a in (r - 1, r) for b in (c - 1, c) if 0 <= a < d and 0 <= b < d]
            inner_r, inner_c = 0 < r < d, 0 < c < d
            if inner_c and (r + c) % 2 == 0 and (inner_r or len(qs) == 2):
                mine.append(qs)
            elif inner_r and (r + c) % 2 == 1 and (inner_c or len(qs) == 2):
                other.append(qs)
    h, l = [0] * (d * d), [0] * (d * d)
    for i, k in enumerate(rng.permutation(len(mine))):
        for x in mine[int(k)]:
            h[x] |= 1 << i
    for r in range(d):
        l[q(r, d // 2)] ^= 1
    for qs in mine:                      # a sum of checks changes no solution's label
        if rng.random() < 0.5:
            for x in qs:
                l[x] ^= 1
    h, l, _ = dedupe(h, l)
    return Problem("surface_d%d" % d, len(mine), 1, h, l, [(i, 0) for i in range(len(mine))])


def _checkpoint(plan, bits):
    """Ops done when the shrinking table last has 2^min(bits, 24) entries: nearly the whole sweep."""
    w, at = 0, 0
    for i, op in enumerate(plan.ops):
        w += 1 if op[0] == "expand" else -1 if op[0] == "select" else 0
        if w == min(bits, 24):
            at = i + 1
    return at, min(bits, 24)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("witness", "distance"):
        s["p"], s["order"], _ = _banded(case, seed, case["nobs"])
    elif kind == "sweep":
        _, _, plans = _banded(case, seed, 1)
        plan = plans[0]
        at, width = _checkpoint(plan, plan.peak_bits)
        s["cp"] = kernel.CompiledPlan(plan, case["dtype"], checkpoints=[at])
        s["a"], s["b"] = s["cp"].buffers()
        s["table"] = device.empty(s["cp"].eb << width)
    elif kind == "batch":
        s["ps"] = synth.batch_instances(seed=seed, count=case["count"], wmin=case["wmin"], wmax=case["wmax"],
                                        max_obs=case["max_obs"])
    elif kind == "tree":
        s["prog"], s["targets"], _ = _tree(case, seed)
        need = s["prog"].preflight(max_join_work=None, max_memory_bytes=None)["device_arena_bytes"]
        s["arena"] = device.empty(need)
    elif kind == "sparse":
        p = synth.circuit_dem(seed=seed, rounds=case["rounds"], checks=case["checks"], ncols=case["ncols"])
        s["tr"] = sparse_dp.plan_trellises(p)[0]
    elif kind == "search":
        s["p"] = _surface(case["d"], seed)
    else:
        rng = np.random.default_rng([seed, 11])
        p = synth.banded(case["m"], case["n"], case["window"], 3, 2, seed=seed)
        s["p"] = p
        zh, zl = search.column_hashes(p.h, search.row_hashes(p.nrows, 12345))
        pick = rng.integers(0, p.ncols, (case["probes"], case["k"] + 1))
        drop = rng.random(pick.shape) < 0.25         # sets of up to k + 1 columns: hits and misses
        at = lambda z: np.bitwise_xor.reduce(np.where(drop, np.uint64(0), z[pick]), axis=1)
        s["zh"], s["zl"] = at(zh), at(zl)
        s["lg"] = rng.integers(0, 4, case["probes"]).astype(np.uint64)
        s["R"] = rng.integers(0, case["k"] + 1, case["probes"]).astype(np.int32)
    return s


# ---------------------------------------------------------------------- one pass
def _value(v):
    return -1 if v is None else int(v)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "witness":
        r = auto.dp_witness(s["p"], s["order"])
        cols = np.zeros(s["p"].ncols, dtype=np.uint8)
        if r is None:
            return {"distance": -1, "observable": -1, "columns": cols}
        cols[r["witness"]] = 1
        return {"distance": r["distance"], "observable": r["observable"], "columns": cols}
    if kind == "distance":
        best, per = auto.dp_distance(s["p"], s["order"])
        return {"best": _value(best), "per": np.array([_value(v) for v in per])}
    if kind == "sweep":
        s["cp"].execute(s["a"], s["b"], [s["table"]])
        return {"entry": s["cp"].result(s["a"], s["b"]), "table": s["table"]}
    if kind == "batch":
        got = batch.batched_dp_distances(s["ps"])
        # the observables of each instance, padded to the most an instance has
        per = np.full((len(got), case["max_obs"]), -2)
        for k, (_, vals) in enumerate(got):
            per[k, :len(vals)] = [_value(v) for v in vals]
        return {"best": np.array([_value(b) for b, _ in got]), "per": per}
    if kind == "tree":
        return {"weights": np.array([_value(s["prog"].run(t, arena=s["arena"], **LIMITS)[0]) for t in s["targets"]])}
    if kind == "sparse":
        r = sparse_dp.query(s["tr"], case["K"])
        return {"value": _value(r["value"]), "peak": int(r["peak_states"]), "forward": np.array(r["forward_counts"]),
                "backward": np.array(r["backward_counts"])}
    if kind == "search":
        r = search.distance(s["p"], k_table=case["k"], kmax=case["d"])
        return {"distance": _value(r["distance"]), "entries": r["table_entries"],
                "nodes": np.array([x["nodes"][0] for x in r["runs"]]),
                "lookups": np.array([x["lookups"] for x in r["runs"]])}
    t = search.Table(s["p"], case["k"])
    out = t.lookup(s["zh"], s["zl"], s["lg"], s["R"])
    t.free()
    return {"entries": t.entries, "costs": out}


# ---------------------------------------------------------------------- what a pass cannot do without
def _subsets(n, k):
    total, c = 0, 1
    for i in range(k + 1):
        total += c
        c = c * (n - i) // (i + 1)
    return total


@functools.lru_cache(maxsize=None)
def _work(items):
    case = dict(items)
    kind = case["kind"]
    if kind in ("witness", "distance", "sweep"):
        nobs = case.get("nobs", 1)
        _, _, plans = _banded(case, 1, nobs)
        updates = sum(pl.work() for pl in plans if pl.feasible)
        eb = 2 if case.get("weights") or case.get("dtype") == "u16" else 1
        out = (eb << min(case["bits"], 24)) if kind == "sweep" else 8 * nobs
        # the columns in, the answers out; an addition and a minimum per state-update
        return 8 * case["n"] * 4 + out, 2 * updates
    if kind == "batch":
        ps = synth.batch_instances(seed=1, count=case["count"], wmin=case["wmin"], wmax=case["wmax"],
                                   max_obs=case["max_obs"])
        updates = sum(pl.work() for p in ps for _, pl in auto._plans(p, list(range(p.ncols))) if pl.feasible)
        return sum(32 * p.ncols + 8 * p.nobs for p in ps), 2 * updates
    if kind == "tree":
        _, targets, work = _tree(case, 1)
        return case["targets"] * (case["n"] // 8 + 4), 2 * work * case["targets"]
    if kind == "sparse":
        # two directions of N columns, each step over tables that grow with K
        return 32 * case["ncols"], 2 * 2 * case["ncols"] * 4 ** case["K"]
    if kind == "search":
        n = case["d"] * case["d"]
        return 9 * 2 * _subsets(n, case["k"]), 2 * _subsets(n, case["k"]) * case["k"]
    subsets = _subsets(case["n"], case["k"])
    return 9 * 2 * subsets + case["probes"] * (8 * 3 + 4 + 4), 2 * subsets * case["k"]


def work(case):
    b, f = _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------- plain numpy
def exact(case, seed):
    """Distances of narrow unit-weight and weighted problems by a plain dynamic programme over the
    parities of the rows that are open in column order (numpy); None for everything else."""
    if case["kind"] not in ("witness", "distance") or case["bits"] > 13:
        return None
    p, order, _ = _banded(case, seed, case["nobs"])
    n = p.ncols
    wt = p.weights or [1] * n
    last = {}
    for j in range(n):
        for r in range(p.nrows):
            if (p.h[j] >> r) & 1:
                last[r] = j
    inf = 1 << 20
    vals = []
    for o in range(p.nobs):
        rows = []                                    # bit k + 1 of a state is rows[k]; bit 0 the logical row
        T = np.array([0, inf], dtype=np.int64)
        for j in range(n):
            m = (p.l[j] >> o) & 1
            for r in [r for r in range(p.nrows) if (p.h[j] >> r) & 1]:
                if r not in rows:
                    rows.append(r)
                    T = np.concatenate([T, np.full(T.size, inf, dtype=np.int64)])
                m |= 2 << rows.index(r)
            if m:
                T = np.minimum(T, T[np.arange(T.size) ^ m] + wt[j])
            for r in [r for r in rows if last[r] == j]:
                k = rows.index(r) + 1
                T = T.reshape(-1, 2, 1 << k)[:, 0].reshape(-1)
                rows.remove(r)
        vals.append(int(T[1]) if T[1] < inf else -1)
    best = min([v for v in vals if v >= 0], default=-1)
    if case["kind"] == "witness":
        return {"distance": best, "observable": None, "columns": None}
    return {"best": best, "per": np.array(vals)}
