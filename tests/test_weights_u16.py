"""Column weights beyond 8 bits on uint16 tables: every form of a pass charges the whole weight (sweeps, tile
passes, granule passes, the one-launch witness).  Whole numbers: results are equal to the oracle's."""
import random

import numpy as np
import pytest

from helpers import emulate
from oracle import dense as od
from tropidist_gb300 import auto, synth, trellis
from tropidist_gb300.kernel import CompiledPlan

DEFAULT = (16, 15, 15, 14)
# (dmax8, dmax16, sweep8, sweep16): sweeps alone, granule passes, tile passes
FORMS = [(16, 15, 15, 15), (16, 15, 15, 9), (16, 10, 15, 9)]
CHOICES = [(1, 255, 256, 257), (1, 1023, 1024, 4095), (3, 32767, 32768, 65534), (254, 511, 16384, 40000)]


@pytest.fixture(autouse=True)
def restore_tuning(lib):
    yield
    lib.tg_dense_set_tuning(*DEFAULT)


def case(seed, form, max_bits):
    rng = random.Random(seed)
    while True:
        m = rng.randint(20, 80)
        n = rng.randint(int(1.3 * m), 3 * m)
        p = synth.banded(m, n, rng.randint(6, 15), rng.choice([2, 3, 4]), 1, seed=rng.randrange(1 << 30))
        p.weights = [rng.choice(CHOICES[seed % len(CHOICES)]) for _ in range(n)]
        plan = trellis.build_plan(p.h, p.l, 1, list(range(n)), p.nrows, weights=p.weights)
        if plan.feasible and (11 if form else 5) <= plan.peak_bits <= max_bits:
            return rng, p, plan


def oracle(plan):
    tabs = []
    try:
        return od.run_plan_numpy(plan, dtype=np.uint16, tables=tabs), tabs
    except OverflowError:
        return 65535, tabs


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("seed", range(8))
def test_emulated_passes_match_oracle(lib, seed, form):
    rng, _, plan = case(seed, form, 14)
    want, tabs = oracle(plan)
    ks = sorted(rng.sample(range(1, len(plan.ops) + 1), min(len(plan.ops), 3)))
    lib.tg_dense_set_tuning(*FORMS[form])
    cp = CompiledPlan(plan, "u16", ks)
    kinds = set(cp.segments()[:, 0].tolist())
    assert (form == 0) == (kinds == {0}) and (form == 1) == (4 in kinds)
    cp.free()
    v, got, _ = emulate(plan, "u16", checkpoints=ks)
    assert v == want
    for k, t in zip(ks, got):
        assert np.array_equal(t, tabs[k - 1])


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("seed", range(4))
def test_kernels_match_oracle(lib, seed, form):
    import torch
    from tropidist_gb300 import device
    from tropidist_gb300.kernel import _width_after
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng, p, plan = case(seed, form, 16 if form else 15)
    want, tabs = oracle(plan)
    ks = sorted(rng.sample(range(1, len(plan.ops) + 1), 3))
    lib.tg_dense_set_tuning(*FORMS[form])
    cp = CompiledPlan(plan, "u16", ks)
    a, b = cp.buffers()
    outs = [device.empty((1 << _width_after(plan.ops, k)) * 2) for k in cp.ckpts]
    cp.execute(a, b, outs)
    assert cp.result(a, b) == want
    for k, o in zip(ks, outs):
        assert np.array_equal(o.cpu().numpy().view(np.uint16), tabs[k - 1])
    cp.free()
    if want == 65535:
        with pytest.raises(OverflowError):
            auto.dp_distance(p, list(range(p.ncols)))
        return
    assert auto.dp_distance(p, list(range(p.ncols)))[0] == want
    w = auto.dp_witness(p, list(range(p.ncols)))
    assert w["distance"] == want == sum(p.weights[j] for j in w["witness"])
