"""Table buffers that are not 16-byte aligned: sweeps and granule passes run on them, a pass that needs
16 bytes refuses them before anything is launched."""
import ctypes

import numpy as np
import pytest

from oracle import dense as od
from tropidist_gb300 import synth, trellis
from tropidist_gb300.kernel import CompiledPlan

DEFAULT = (16, 15, 15, 14)
TG_ERR_ARG = -1


def plan_of(m, n, window, seed=0):
    p = synth.banded(m, n, window, 3, 1, seed=seed)
    return trellis.build_plan(p.h, p.l, 1, list(range(n)), p.nrows)


@pytest.fixture(autouse=True)
def restore_tuning(lib):
    yield
    lib.tg_dense_set_tuning(*DEFAULT)


@pytest.mark.parametrize("dtype,off", [("u8", 4), ("u8", 8), ("u16", 2), ("u16", 8)])
def test_passes_that_need_aligned_buffers_refuse_others(lib, dtype, off):
    """The refusal needs no device: the addresses are never used."""
    lib.tg_dense_set_tuning(10, 10, 9, 9)              # tile passes and no granule passes
    plan = plan_of(120, 240, 14)
    cp = CompiledPlan(plan, dtype)
    assert set(cp.segments()[:, 0]) & {1, 3}
    a, b, out = 1 << 20, 1 << 21, (ctypes.c_double * 15)()
    for x, y in ((a + off, b), (a, b + off)):
        assert lib.tg_dense_execute(cp.handle, x, y, None, None) == TG_ERR_ARG
        assert lib.tg_dense_execute_timed(cp.handle, x, y, None, out, 15) == TG_ERR_ARG
    cp.free()


@pytest.mark.gpu
@pytest.mark.parametrize("window", [8, 15, 18])
@pytest.mark.parametrize("dtype", ["u8", "u16"])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 5, 8])
def test_plans_run_on_unaligned_buffers(lib, window, dtype, shift):
    """Sweeps (narrow plans) on buffers of any alignment, granule passes on 4-byte aligned ones; one
    checkpoint in a buffer of its own alignment."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    plan = plan_of(120, 240, window, seed=window)
    tabs = []
    want = od.run_plan_numpy(plan, dtype=np.uint8 if dtype == "u8" else np.uint16, tables=tabs)
    k = len(plan.ops) // 2
    cp = CompiledPlan(plan, dtype, [k])
    kinds = set(cp.segments()[:, 0].tolist())
    assert kinds <= {0, 1, 4} and ((4 in kinds) == (window == 18))
    off = shift * cp.eb
    n = (1 << cp.peak_bits) * cp.eb
    mem = torch.full((3, n + 256), 85, dtype=torch.uint8, device="cuda")
    a, b, o = mem[0, off:off + n], mem[1, 3 * off:3 * off + n], mem[2, off:off + tabs[k - 1].nbytes]
    if kinds == {0} or off % 16 == 0 or (1 not in kinds and off % 4 == 0):
        cp.execute(a, b, [o])
        assert cp.result(a, b) == want
        assert np.array_equal(o.cpu().numpy().view(tabs[k - 1].dtype), tabs[k - 1])
        for t, x in ((mem[0], off), (mem[1], 3 * off)):            # nothing outside the tables
            assert bool((t[:x] == 85).all()) and bool((t[x + n:] == 85).all())
    else:
        assert lib.tg_dense_execute(cp.handle, a.data_ptr(), b.data_ptr(), None, None) == TG_ERR_ARG
    cp.free()
