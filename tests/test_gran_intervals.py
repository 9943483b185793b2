"""Granule passes between kept tables: taken by the number of ops between two of them and the width there,
interval by interval, with equal tables whichever form takes an interval."""
import random

import numpy as np
import pytest

from helpers import emulate
from oracle import dense as od
from tropidist_gb300 import synth, trellis
from tropidist_gb300.kernel import CompiledPlan

DEFAULT = (16, 15, 15, 14)


@pytest.fixture(autouse=True)
def restore_tuning(lib):
    yield
    lib.tg_dense_set_tuning(*DEFAULT)


def plan_of(window, seed=0):
    p = synth.banded(150, 300, window, 3, 1, seed=seed)
    return trellis.build_plan(p.h, p.l, 1, list(range(300)), p.nrows)


def wide_segments(plan, dtype, ks, bits, ops=(0, 1 << 60)):
    """Forms of the segments on tables of `bits` bits or more that end within the ops given."""
    cp = CompiledPlan(plan, dtype, ks)
    s = cp.segments()
    cp.free()
    return [int(x[0]) for x in s if min(x[1], x[2]) >= bits and ops[0] < x[3] <= ops[1]]


def flat_plan(width, updates=240):
    """`updates` columns on a table of constant width."""
    rng = random.Random(width)
    ops = [("expand",)] * width
    ops += [("update", sum(1 << q for q in rng.sample(range(width), 3)), 1) for _ in range(updates)]
    return trellis.Plan(ops + [("select", 0, 0)] * width, width, [], 0)


@pytest.mark.parametrize("width,dtype,every,gran", [
    (17, "u8", 3, False), (17, "u8", 4, True), (20, "u8", 7, False), (24, "u8", 7, False), (24, "u8", 8, True),
    (25, "u8", 9, False), (25, "u8", 10, True), (27, "u8", 13, False), (27, "u8", 14, True), (30, "u8", 15, False),
    (30, "u8", 16, True), (23, "u16", 8, False), (23, "u16", 9, True), (24, "u16", 5, False), (30, "u16", 6, True)])
def test_fewest_ops_between_kept_tables(width, dtype, every, gran):
    plan = flat_plan(width)
    last = width + 240 // every * every
    forms = wide_segments(plan, dtype, list(range(width, last + 1, every)), width, (width, last - 1))
    assert len(forms) > 10 and (4 in forms) == gran


def test_one_bunch_of_kept_tables_leaves_the_rest_of_the_plan():
    plan = plan_of(26)
    n = len(plan.ops)
    bunch = list(range(n // 2, n // 2 + 100))
    assert 4 not in wide_segments(plan, "u8", bunch, 20, (n // 2, n // 2 + 99))
    for span in ((0, n // 2), (n // 2 + 99, n)):
        assert 4 in wide_segments(plan, "u8", bunch, 20, span)


@pytest.mark.parametrize("seed", range(6))
def test_tables_kept_at_random_gaps_match_oracle(lib, seed):
    rng = random.Random(seed)
    p = synth.banded(60, 130, 16, 3, 1, seed=seed)
    plan = trellis.build_plan(p.h, p.l, 1, list(range(p.ncols)), p.nrows)
    tabs = []
    for dtype, npd in (("u8", np.uint8), ("u16", np.uint16)):
        lib.tg_dense_set_tuning(16, 15, 9, 9)
        ks, k = [], 0
        while True:
            k += rng.choice([1, 1, 3, 5, 8, 12, 20])
            if k > len(plan.ops):
                break
            ks.append(k)
        tabs = []
        want = od.run_plan_numpy(plan, dtype=npd, tables=tabs)
        v, got, _ = emulate(plan, dtype, checkpoints=ks)
        assert v == want
        for k, t in zip(ks, got):
            assert np.array_equal(t, tabs[k - 1])
