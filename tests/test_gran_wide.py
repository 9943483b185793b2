"""Granule passes of tables near and beyond 2^32 granules (csrc/gran_sched.h): their offsets are 32-bit
granule numbers, so wider tables take the forms with 64-bit offsets.  Only schedules are built: no table
is allocated."""
import numpy as np
import pytest

from tropidist_gb300 import synth, trellis
from tropidist_gb300.kernel import CompiledPlan


def rank(vectors):
    basis = {}
    for v in vectors:
        v = int(v)
        while v:
            t = v.bit_length()
            if t not in basis:
                basis[t] = v
                break
            v ^= basis[t]
    return len(basis)


def gran_maps(lib, cp, seg):
    m, n = np.zeros((2, 40), dtype=np.uint32), np.zeros(2, dtype=np.int32)
    assert lib.tg_debug_gran_maps(cp.handle, seg, m[0].ctypes.data, m[1].ctypes.data, n.ctypes.data) == 0
    return m[0, :n[0]].tolist(), m[1, :n[1]].tolist()


# (m, n, window, column weight, entry type): peaks of 33 to 38 bits
PLANS = [(200, 400, 38, 3, "u8"), (200, 400, 38, 3, "u16"), (200, 400, 40, 3, "u8"), (200, 400, 40, 3, "u16"),
         (200, 400, 42, 3, "u8"), (200, 400, 42, 3, "u16"), (1000, 2000, 42, 3, "u16"), (1000, 2000, 44, 3, "u8"),
         (400, 800, 38, 5, "u8"), (400, 800, 38, 5, "u16")]


@pytest.mark.parametrize("m,n,window,weight,dtype", PLANS)
def test_every_granule_has_one_address(lib, m, n, window, weight, dtype):
    """The offsets of a pass's coset bits and slots are independent on both sides, and no granule pass
    reads or writes a table of more than 2^32 granules."""
    p = synth.banded(m, n, window, weight, 1, seed=0)
    plan = trellis.build_plan(p.h, p.l, 1, list(range(n)), p.nrows)
    assert plan.feasible and plan.peak_bits >= 31
    cp = CompiledPlan(plan, dtype)
    per = 2 if cp.eb == 1 else 1          # entries per granule (log2)
    passes = 0
    for k, s in enumerate(cp.segments()):
        if s[0] != 4:
            continue
        passes += 1
        assert max(s[1], s[2]) <= 32 + per
        vin, vout = gran_maps(lib, cp, k)
        assert rank(vin) == len(vin) and rank(vout) == len(vout) == s[2] - per
    cp.free()
    assert passes > 10
