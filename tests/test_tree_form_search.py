"""Block-product forms are looked for only on joins that could run as one."""
import pytest

from tropidist_gb300 import synth, tree_dp


def balanced(cols):
    if len(cols) == 1:
        return cols[0]
    h = len(cols) // 2
    return (balanced(cols[:h]), balanced(cols[h:]))


@pytest.mark.parametrize("m,n,window", [(45, 90, 8), (80, 160, 10), (120, 240, 12)])
def test_forms_looked_for(m, n, window, monkeypatch):
    prog = tree_dp.CompiledTreeDP(synth.banded(m, n, window, 3, 1, seed=0).h, balanced(list(range(n))))
    form, asked = tree_dp.gemm_form, []
    monkeypatch.setattr(tree_dp, "gemm_form", lambda jn: asked.append(jn) or form(jn))
    prog.preflight()
    for jn in asked:
        F = len(jn.free_maps)
        assert F >= 2 and min(jn.left_rank, jn.right_rank) >= F + 6
    # nothing that runs is among the others
    for jn in prog.joins.values():
        g = form(jn)
        assert any(jn is a for a in asked) or g is None or not tree_dp.runs_as_product(g)
    assert len(asked) < len(prog.joins) / 2
