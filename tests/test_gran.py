"""Granule passes (csrc/gran.cuh): the scheduler's register programs and address maps through the host
emulation, and the kernel on the GPU, against the oracle's tables at checkpoints.  Low sweep limits make
the passes run from 9-bit tables up, where rows open and close every few columns, lanes outnumber the
free rows and the in-granule rows change places in almost every pass.  Results are whole numbers and
must be equal."""
import random

import numpy as np
import pytest

from helpers import emulate
from oracle import dense as od
from tropidist_gb300 import synth, trellis

DEFAULT = (16, 15, 15, 14)


@pytest.fixture(autouse=True)
def restore_tuning(lib):
    yield
    lib.tg_dense_set_tuning(*DEFAULT)
    lib.tg_dense_set_stream_span(3, 2)


def cases(seed, count, max_bits):
    """Random banded plans with their dtype, checkpoints and the oracle's value and tables."""
    rng = random.Random(seed)
    found = 0
    while found < count:
        m = rng.randint(20, 120)
        n = rng.randint(int(1.3 * m), 3 * m)
        p = synth.banded(m, n, rng.randint(9, 18), rng.choice([2, 3, 3, 4, 5]), 1, seed=rng.randrange(1 << 30))
        w = [rng.choice([1, 2, 3, 100, 253]) for _ in range(n)] if rng.random() < 0.5 else None
        plan = trellis.build_plan(p.h, p.l, 1, list(range(n)), p.nrows, weights=w)
        if not plan.feasible or not 11 <= plan.peak_bits <= max_bits:
            continue
        found += 1
        for dtype, npd, inf in (("u8", np.uint8, 255), ("u16", np.uint16, 65535)):
            tune = (rng.choice([12, 16]), rng.choice([9, 10, 12]), rng.choice([11, 15]), rng.choice([9, 10, 12]))
            ks = sorted(rng.sample(range(1, len(plan.ops) + 1), min(len(plan.ops), rng.randint(0, 3))))
            tabs = []
            try:
                want = od.run_plan_numpy(plan, dtype=npd, tables=tabs)
            except OverflowError:
                want = inf
            yield plan, dtype, tune, ks, inf if want is None else want, [tabs[k - 1] for k in ks]


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_emulated_passes_match_oracle(lib, seed):
    from tropidist_gb300.kernel import CompiledPlan
    passes = 0
    for plan, dtype, tune, ks, want, want_tabs in cases(seed, 10, 16):
        lib.tg_dense_set_tuning(*tune)
        v, tabs, _ = emulate(plan, dtype, checkpoints=ks)
        assert v == want
        for a, b in zip(tabs, want_tabs):
            assert np.array_equal(a, b)
        cp = CompiledPlan(plan, dtype, ks)
        passes += int((cp.segments()[:, 0] == 4).sum())
        cp.free()
    assert passes > 10


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [11, 12])
def test_kernel_matches_oracle(lib, seed):
    import torch
    from tropidist_gb300 import device
    from tropidist_gb300.kernel import CompiledPlan, _width_after
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    for plan, dtype, tune, ks, want, want_tabs in cases(seed, 12, 18):
        lib.tg_dense_set_tuning(*tune)
        cp = CompiledPlan(plan, dtype, ks)
        a, b = cp.buffers()
        outs = [device.empty((1 << _width_after(plan.ops, k)) * cp.eb) for k in cp.ckpts]
        cp.execute(a, b, outs)
        assert cp.result(a, b) == want
        for o, t in zip(outs, want_tabs):
            assert np.array_equal(o.cpu().numpy().view(t.dtype), t)
        cp.free()


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [3, 4])
def test_batched_passes_match_single(lib, seed):
    """The same passes as units of the persistent kernel: the final entries of plans of 12 to 20 bits."""
    import torch
    from tropidist_gb300 import auto, kernel
    from tropidist_gb300.batch import DenseBatch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    ps = synth.batch_instances(seed=seed, count=6, wmin=12, wmax=20, max_obs=3)
    plans = [pl for p in ps for _, pl in auto._plans(p, list(range(p.ncols)))]
    got = DenseBatch(plans).run()
    for pl, v in zip(plans, got):
        assert v == (kernel.run_plan(pl)[0] if pl.feasible else None)


@pytest.mark.parametrize("every,gran", [(1, False), (3, False), (4, True), (16, True)])
def test_checkpoints_every_few_ops_take_the_other_forms(every, gran):
    """A granule pass between checkpoints an op or two apart would hold one column."""
    from tropidist_gb300 import kernel
    p = synth.banded(120, 300, 18, 3, 1, seed=3)
    plan = trellis.build_plan(p.h, p.l, 1, list(range(300)), p.nrows)
    cp = kernel.CompiledPlan(plan, "u8", list(range(every, len(plan.ops), every)))
    assert (4 in cp.segments()[:, 0]) == gran
    cp.free()
