"""The persistent kernels' two kinds: the one without the fast forms of tile and streaming passes takes a
stray such pass tile by tile, the other is chosen by the table bytes that the passes of each kind move.
Values against the oracle's tables, the kinds by the library's own account of them."""
import random
import time

import numpy as np
import pytest

from oracle import dense as od
from tropidist_gb300 import synth, trellis

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DEFAULT = (16, 15, 15, 14)


@pytest.fixture(autouse=True)
def knobs(lib):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    yield
    lib.tg_dense_set_tuning(*DEFAULT)
    lib.tg_dense_set_stream_span(3, 2)


def with_stray_passes(seed, count, window=19):
    """A banded plan with `count` places where two rows open, a column uses both, and two rows close."""
    rng = random.Random(seed)
    while True:
        p = synth.banded(90, 180, window - rng.randint(0, 2), 3, 1, seed=rng.randrange(1 << 30))
        weights = [rng.randint(1, 9) for _ in range(p.ncols)]
        plan = trellis.build_plan(p.h, p.l, 1, list(range(p.ncols)), p.nrows, weights=weights)
        w, at = 0, []
        for k, op in enumerate(plan.ops):
            if op[0] == "update" and w >= 15:
                at.append((k, w))
            w += {"expand": 1, "update": 0, "select": -1}[op[0]]
        if plan.feasible and len(at) > 2 * count and window - 3 <= plan.peak_bits <= window - 1:
            break
    ops = list(plan.ops)
    for k, w in sorted(rng.sample(at, count), reverse=True):
        ops[k:k] = [("expand",), ("expand",), ("update", 3 << w | rng.getrandbits(w), rng.choice([1, 2])),
                    ("select", w + 1, 0), ("select", w, 0)]
    return trellis.Plan(ops, plan.peak_bits + 2, [], 0)


def test_stray_passes_in_the_kernel_without_their_fast_forms(lib):
    from tropidist_gb300.batch import DenseBatch
    plans = [with_stray_passes(s, 1 + s % 2) for s in range(5)] + [with_stray_passes(s, 0, 22) for s in range(3)]
    want = [od.run_plan_numpy(pl) for pl in plans]
    b = DenseBatch(plans)
    info = np.zeros(7, dtype=np.int64)
    assert lib.tg_batch_info(b.handle, info.ctypes.data, 7) == 0
    gran, other, fast = info[4:].tolist()
    assert other > 0 and 4 * other <= gran and not fast
    for _ in range(2):
        assert b.run() == want


@pytest.mark.parametrize("tune,span", [(DEFAULT, (3, 3)), ((11, 15, 10, 14), (3, 2))])
def test_batches_of_other_passes_take_the_kernel_with_them(lib, tune, span):
    from tropidist_gb300.batch import DenseBatch
    lib.tg_dense_set_tuning(*tune)
    lib.tg_dense_set_stream_span(*span)
    plans = [with_stray_passes(s, 2) for s in range(6)]
    b = DenseBatch(plans)
    info = np.zeros(7, dtype=np.int64)
    assert lib.tg_batch_info(b.handle, info.ctypes.data, 7) == 0
    assert info[4] == 0 and info[5] > 0 and info[6] == 1
    assert b.run() == [od.run_plan_numpy(pl) for pl in plans]


def test_server_chooses_by_the_plans_in_progress(lib):
    """A plan of other passes does not settle the kernel of later plans."""
    import ctypes
    from tropidist_gb300.kernel import CompiledPlan
    plan = with_stray_passes(1, 0)
    want = od.run_plan_numpy(plan)
    gran = CompiledPlan(plan, "u8")
    lib.tg_dense_set_stream_span(3, 3)
    other = CompiledPlan(plan, "u8")
    assert 4 in gran.segments()[:, 0] and 4 not in other.segments()[:, 0]
    arena = torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    st = ctypes.c_int(0)
    srv = lib.tg_server_create(arena.data_ptr(), arena.numel(), 1 << 12, 1 << 24, 16, 8, ctypes.byref(st))
    assert srv and st.value == 0
    slots, vals = np.zeros(16, dtype=np.int32), np.zeros(16, dtype=np.uint32)

    def done():
        for _ in range(20000):
            n = lib.tg_server_poll(srv, slots.ctypes.data, vals.ctypes.data, 16)
            assert n >= 0
            if n:
                return vals[:n].tolist()
            time.sleep(1e-4)
        raise AssertionError("no result within two seconds")

    try:
        assert lib.tg_server_form(srv) == 0
        for cp, form in ((gran, 0), (other, 1), (gran, 0)):
            assert lib.tg_server_submit_plan(srv, cp.handle) >= 0
            assert lib.tg_server_form(srv) == form
            assert done() == [want]
        assert lib.tg_server_form(srv) == 0
    finally:
        lib.tg_server_free(srv)
        gran.free()
        other.free()
