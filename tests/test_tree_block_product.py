"""The block-product form of tree joins whose parents do not cover every pair of child blocks: the identity
of the maps on the CPU, and k_tree_gemm with row maps against the per-pair kernel and the oracle."""
import random

import pytest
import torch

from oracle import tree as ot
from tropidist_gb300 import synth, tree_dp

gpu = pytest.mark.gpu


def balanced(cols):
    if len(cols) == 1:
        return cols[0]
    h = len(cols) // 2
    return (balanced(cols[:h]), balanced(cols[h:]))


def xor(vectors, x):
    out = 0
    for i, v in enumerate(vectors):
        if x >> i & 1:
            out ^= v
    return out


def coupled(prog):
    """Joins with a block product whose blocks do not all meet, as (join, form)."""
    out = []
    for jn in prog.joins.values():
        g = tree_dp.gemm_form(jn)
        if g is not None and g["mb"] + g["nb"] < jn.left_rank + jn.right_rank - 2 * g["F"]:
            out.append((jn, g))
    return out


@pytest.mark.parametrize("m,n,win,seed", [(30, 60, 8, 0), (41, 83, 9, 1), (64, 125, 12, 2), (80, 160, 10, 2)])
def test_form_reproduces_the_maps(m, n, win, seed):
    prog = tree_dp.CompiledTreeDP(synth.banded(m, n, win, 3, 1, seed=seed).h, balanced(list(range(n))))
    rng = random.Random(seed)
    seen = 0
    for jn in prog.joins.values():
        g = tree_dp.gemm_form(jn)
        if g is None:
            continue
        seen += 1
        F, lr = g["F"], jn.left_rank
        e = tree_dp._Eliminator()
        for v in g["PA"] + g["PB"] + g["PT"]:
            e.add(v)
        assert e.rank() == jn.parent_rank == g["mb"] + g["nb"] + g["kb"]
        for _ in range(20):
            x, y, t = (rng.randrange(1 << g[k]) for k in ("mb", "nb", "kb"))
            p = xor(g["PA"], x) ^ xor(g["PB"], y) ^ xor(g["PT"], t)
            s = xor(list(jn.parent_maps), p)
            left, right = s & ((1 << lr) - 1), s >> lr
            assert left == (xor(g["GA"], x) ^ xor(g["TA"], t)) << F
            assert right >> F == xor(g["GB"], y) ^ xor(g["TB"], t)
            assert right & ((1 << F) - 1) == xor(g["DL"], x) ^ xor(g["DR"], y) ^ xor(g["DT"], t)
    assert seen and coupled(prog)


@gpu
@pytest.mark.parametrize("m,n,win,seed,check", [
    (70, 140, 11, 1, "oracle"), (80, 160, 12, 1, "oracle"), (90, 180, 11, 4, "device"),
    (101, 203, 12, 9, "device"), (120, 240, 12, 2, "device"), (120, 240, 12, 5, "device")])
def test_row_maps_on_the_device(m, n, win, seed, check):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    prog = tree_dp.CompiledTreeDP(synth.banded(m, n, win, 3, 1, seed=seed).h, balanced(list(range(n))))
    assert any(g["F"] >= 2 and min(g["mb"], g["nb"]) >= 6 for _, g in coupled(prog))
    lim = dict(max_join_work=None, max_memory_bytes=None, max_seconds=None)
    rng = random.Random(seed)
    for t in [rng.randrange(1 << m) for _ in range(3)]:
        got = prog.run(t, **lim)[0]
        want = ot.run(prog, t) if check == "oracle" else prog.run(t, gemm=False, **lim)[0]
        assert got == want
    prog.free()
