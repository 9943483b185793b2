"""Completion tables of problems with few distinct keys (most subsets meet a key that is there already), on both
sides of the rule that reads a slot before claiming it: entries and probes against the enumeration oracle."""
import random

import pytest

from oracle import table as ot
from tropidist_gb300 import search
from tropidist_gb300.problem import Problem

pytestmark = pytest.mark.gpu


# subsets 2^15 (rule: rank 8), 2^13 (rank 6), 2^20.2 (rank 15); at most m + nobs independent keys
@pytest.mark.parametrize("n,k,m,nobs", [(60, 3, 1, 1), (60, 3, 3, 2), (60, 3, 6, 2), (60, 3, 7, 2), (60, 3, 30, 2),
                                        (120, 2, 4, 2), (120, 2, 5, 2), (188, 3, 12, 3), (188, 3, 14, 3)])
@pytest.mark.parametrize("labelfree", [False, True])
def test_entries_and_probes(n, k, m, nobs, labelfree):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = random.Random(n + m)
    h = [rng.randrange(1, 1 << m) for _ in range(n)]
    p = Problem("few", m, nobs, h, [rng.randrange(1 << nobs) for _ in range(n)])
    T = search.Table(p, k, labelfree=labelfree)
    ent = ot.entries(T.zh, T.zl, T.lg, k)
    assert T.entries == len(ent)
    syn = [rng.randrange(1 << m) for _ in range(200)]
    lab = [1 if labelfree else rng.randrange(1 << nobs) for _ in range(200)]
    zh, zl = T.hashes_for(syn)
    for R in range(k + 1):
        want = [ot.lookup(ent, zl[i], lab[i], R) for i in range(len(syn))]
        assert T.lookup_syndromes(syn, lab, R).tolist() == want
    T.free()
