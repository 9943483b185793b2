"""Trees with tables beyond the device's 32-bit state index: they are accounted for and refused, and their
joins take no block-product form (whose maps are 32-bit)."""
import pytest

from tropidist_gb300 import synth, tree_dp


def balanced(cols):
    if len(cols) == 1:
        return cols[0]
    h = len(cols) // 2
    return (balanced(cols[:h]), balanced(cols[h:]))


@pytest.mark.parametrize("m,n,window,seed", [(150, 300, 30, 0), (150, 300, 30, 1), (200, 400, 36, 0), (200, 400, 40, 1)])
def test_wide_trees_are_accounted_for_and_refused(m, n, window, seed, monkeypatch):
    p = synth.banded(m, n, window, 3, 1, seed=seed)
    prog = tree_dp.CompiledTreeDP(p.h, balanced(list(range(n))))
    assert max(jn.parent_rank for jn in prog.joins.values()) > tree_dp.DEVICE_INDEX_BITS
    pf = prog.preflight(max_memory_bytes=None, max_join_work=None)
    with pytest.raises(tree_dp.TreeDPResourceError):
        prog.run(0)
    with pytest.raises(tree_dp.TreeDPResourceError):
        prog.device_plan()
    # the accounting does not depend on the forms of the joins
    plain = tree_dp.CompiledTreeDP(p.h, balanced(list(range(n))))
    monkeypatch.setattr(tree_dp, "gemm_form", lambda jn: None)
    want = plain.preflight(max_memory_bytes=None, max_join_work=None)
    same = lambda d: {k: v for k, v in d.items() if "seconds" not in k}
    assert same(pf) == same(want)
