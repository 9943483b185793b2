"""The one-launch witness of small plans (tables in shared memory up to 2^17 bytes, beyond that through L2)
against the traceback by checkpoints and bisection: both walk back by the same rule, so the columns are
the same."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,window,weighted,bits", [
    (6, 13, 6, False, 0),            # tables below one 16-byte chunk
    (40, 80, 10, False, 0),
    (120, 240, 16, False, 14),
    (120, 241, 18, True, 15),        # uint16
    (90, 180, 19, False, 16),        # 2^17 bytes and beyond
    (80, 160, 21, False, 18),
    (90, 180, 19, True, 16),
])
def test_small_witness_equals_bisection(m, n, window, weighted, bits, monkeypatch):
    from tropidist_gb300 import auto, synth
    from tropidist_gb300.problem import verify_witness
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    for seed in range(3):
        p = synth.banded(m, n, window, 3, 2, seed=seed)
        if weighted:
            p.weights = [1 + (7 * j + seed) % 3 for j in range(p.ncols)]
        order = list(range(p.ncols))
        assert max(pl.peak_bits for _, pl in auto._plans(p, order)) >= bits
        got = {}
        for small in (256 << 20, 0):
            monkeypatch.setattr(auto, "SMALL_WITNESS_BYTES", small)
            got[small] = auto.dp_witness(p, order)
        a, b = got[256 << 20], got[0]
        assert a == b
        if a is not None:
            assert verify_witness(p, a["witness"], a["observable"])
