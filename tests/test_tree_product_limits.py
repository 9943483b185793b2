"""The sizes of tree joins that run as block products: within the launch grid of k_tree_gemm."""
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest

from tropidist_gb300 import tree_dp

TG_ERR_ARG = -1


def coupled_join(mb, nb, kb, F=2):
    """A join of 2^mb left and 2^nb right rows of its own and kb couplings of a left and a right row."""
    left, right = F + mb + kb, F + nb + kb
    gen = lambda a, b: (a << F) | (b << F) << left
    maps = [gen(1 << i, 0) for i in range(mb)] + [gen(0, 1 << i) for i in range(nb)]
    maps += [gen(1 << (mb + i), 1 << (nb + i)) for i in range(kb)]
    return SimpleNamespace(left_rank=left, right_rank=right, parent_rank=len(maps), parent_maps=maps,
                           free_maps=[(1 << k) | (1 << k) << left for k in range(F)])


def plan_status(lib, jn, g):
    """tg_tree_plan's status for this one join as a block product (2: a refusal of the row itself)."""
    F, P = g["F"], jn.parent_rank
    lo, ro, po = 0, 1 << jn.left_rank, (1 << jn.left_rank) + (1 << jn.right_rank)
    arena = po + (1 << P)
    leaves = np.array([[lo, 1, 0, 0], [ro, 1, 1, 0]], dtype=np.int64)
    joins = np.array([[lo, ro, po, P, F, 1, 0, 0]], dtype=np.int64)
    lm = (1 << jn.left_rank) - 1
    maps = np.array([[m & lm, m >> jn.left_rank] for m in jn.parent_maps + jn.free_maps], dtype=np.uint32)
    gmaps = np.array(sum((g[k] for k in ("DL", "DR", "DT", "PA", "PB", "PT", "GA", "GB", "TA", "TB")), []), dtype=np.uint32)
    row = np.array([[0, F | tree_dp.GEMM_ROWS, g["mb"], g["nb"], g["kb"], 0]], dtype=np.int64)
    st = ctypes.c_int(0)
    h = lib.tg_tree_plan(leaves.ctypes.data, 2, joins.ctypes.data, 1, maps.ctypes.data, len(maps), row.ctypes.data, 1,
                         gmaps.ctypes.data, len(gmaps), arena, po, 2, -1, -1, ctypes.byref(st))
    msg = lib.tg_last_error().decode() if not h else ""
    if h:
        lib.tg_tree_plan_free(h)
    return 2 if st.value == TG_ERR_ARG and "gemm" in msg else 0


@pytest.mark.parametrize("kb,runs", [(0, True), (1, True), (14, True), (15, True), (16, False), (17, False)])
def test_products_fit_the_launch_grid(lib, kb, runs):
    jn = coupled_join(6, 6, kb)
    g = tree_dp.gemm_form(jn)
    assert (g["mb"], g["nb"], g["kb"]) == (6, 6, kb)
    assert tree_dp.runs_as_product(g) == runs == (1 << kb <= 65535)
    assert (plan_status(lib, jn, g) == 0) == runs
