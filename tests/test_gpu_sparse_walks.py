"""Sparse walks across their table-size regimes (shared memory, one block on the global scratch, separate
kernels) and the one-launch traceback, against the oracle's tables and queries: problems whose tables
cross 2048 and 8192 states (154083 backwards), with and without lookahead, falling caps (truncated tables) and kept tables
at every cut.  Whole numbers: equal."""
import pytest

from oracle.sparse import NumpyTables
from oracle.sparse_wide import WideTables

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def _trellis(seed, rounds, checks, ncols):
    from tropidist_gb300 import sparse_dp, synth
    p = synth.circuit_dem(seed=seed, rounds=rounds, checks=checks, ncols=ncols)
    return p, sparse_dp.Trellis.for_query(p, 0, sparse_dp.default_order(p))


def _tables(be, tab):
    keys, vals = be.arrays(tab)
    return [int(k) for k in keys], [int(v) for v in vals]


@pytest.mark.parametrize("checks,ncols,K,use_h,peak", [(20, 500, 5, True, 0),
                                                        (18, 400, 5, False, 2048)])
@pytest.mark.parametrize("direction", [+1, -1])
def test_sweeps_match_oracle(direction, checks, ncols, K, use_h, peak):
    from tropidist_gb300 import sparse_dp
    p, tr = _trellis(3, 4, checks, ncols)
    assert tr.nslots <= 56
    g = sparse_dp.Sweep(tr, direction, K, K, use_h=use_h, every=9)
    g.run()
    o = sparse_dp.Sweep(tr, direction, K, K, use_h=use_h, every=9, backend=NumpyTables(tr))
    o.run(on_cut=lambda *a: False)
    assert g.counts == o.counts and g.peak == o.peak and g.peak >= peak
    for c, t in g.ckpt.items():
        assert _tables(g.be, t) == _tables(o.be, o.ckpt[c]), c


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("seed,K", [(1, 4), (2, 7)])
def test_queries_and_witnesses_match_oracle(wide, seed, K):
    """The meet in the middle by walks and the traceback in one launch per interval: value, peak and
    changed counts of the oracle's step-by-step meet; the witness is a solution of that weight."""
    from tropidist_gb300 import sparse_dp
    p, tr = _trellis(seed, 4, 90 if wide else 18, 900 if wide else 500)
    assert (tr.nslots > 64) == wide
    got = sparse_dp.query(tr, K)
    want = sparse_dp.query(tr, K, backend=WideTables(tr) if wide else NumpyTables(tr))
    for k in ("value", "peak_states", "changed_counts", "forward_counts", "backward_counts"):
        assert got[k] == want[k], k
    if got["value"] is not None:
        s = lg = 0
        for j in got["witness"]:
            s ^= p.h[j]
            lg ^= p.l[j]
        assert s == 0 and lg & 1 and sum(p.weights[j] for j in got["witness"]) == got["value"]
