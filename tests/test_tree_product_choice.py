"""Which joins of a tree run as block products: with couplings between left and right rows from 2^22 pairs on,
where every left block meets every right block as soon as the form runs."""
import pytest

from tropidist_gb300 import synth, tree_dp


def balanced(cols):
    if len(cols) == 1:
        return cols[0]
    h = len(cols) // 2
    return (balanced(cols[:h]), balanced(cols[h:]))


@pytest.mark.parametrize("m,n,window", [(60, 120, 9), (80, 160, 10), (80, 160, 12), (100, 200, 12), (120, 240, 12),
                                        (150, 300, 10)])
def test_small_coupled_joins_stay_with_the_pairs(m, n, window):
    left_out = taken = 0
    for seed in range(3):
        prog = tree_dp.CompiledTreeDP(synth.banded(m, n, window, 3, 1, seed=seed).h, balanced(list(range(n))))
        lay = prog._layout()
        products = set(lay["gemm"][:, 0].tolist())
        # the layout's rows are the joins by height and node
        height = {}
        for i, nd in enumerate(prog.nodes):
            height[i] = 0 if nd.leaf is not None else 1 + max(height[nd.left], height[nd.right])
        order = sorted((i for i in height if height[i]), key=lambda i: (height[i], i))
        assert len(order) == len(lay["joins"])
        for row, i in enumerate(order):
            jn = prog.joins[i]
            g = tree_dp.gemm_form(jn)
            runs = g is not None and g["F"] >= 2 and 6 <= g["mb"] <= 21 and 6 <= g["nb"] <= 21 and g["kb"] <= 15
            coupled = runs and g["mb"] + g["nb"] < jn.left_rank + jn.right_rank - 2 * g["F"]
            small = jn.parent_rank + len(jn.free_maps) < 22
            assert (row in products) == (runs and not (coupled and small))
            left_out += coupled and small
            taken += coupled and not small
    assert left_out if window < 12 else taken
