"""Wide sparse walks across their regimes (shared memory, one block on L2 scratch, separate launches) with
states of two to six words, against the oracle's tables.  Whole numbers: equal."""
import pytest

from oracle.sparse_wide import WideTables

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# peaks 1932, 1744, 602 and 1445 states backwards: past the shared tables' 512 (256 from five words up)
@pytest.mark.parametrize("words,seed,rounds,checks,ncols,K", [(2, 1, 4, 150, 900, 5), (3, 2, 3, 300, 1200, 5),
                                                              (4, 1, 4, 500, 2500, 4), (6, 1, 4, 700, 4000, 4)])
@pytest.mark.parametrize("limit", [None, 600, 0])
def test_walks_match_oracle(words, seed, rounds, checks, ncols, K, limit):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from tropidist_gb300 import _lib, sparse_dp, synth
    L = _lib.lib()
    p = synth.circuit_dem(seed=seed, rounds=rounds, checks=checks, ncols=ncols)
    tr = sparse_dp.Trellis.for_query(p, 0, sparse_dp.default_order(p))
    assert (tr.nslots + 63) // 64 == words
    old = L.tg_spw_set_small_limit(-1)
    try:
        if limit is not None:
            L.tg_spw_set_small_limit(limit)
        for direction in (+1, -1):
            g = sparse_dp.Sweep(tr, direction, K, K, use_h=True, every=9)
            g.run()
            o = sparse_dp.Sweep(tr, direction, K, K, use_h=True, every=9, backend=WideTables(tr))
            o.run(on_cut=lambda *a: False)
            assert g.counts == o.counts and g.peak == o.peak
            assert direction > 0 or g.peak > 512
            for c, t in g.ckpt.items():
                (gk, gv), (ok, ov) = g.be.arrays(t), o.be.arrays(o.ckpt[c])
                assert [int(x) for x in gk] == [int(x) for x in ok] and list(map(int, gv)) == list(map(int, ov)), c
    finally:
        L.tg_spw_set_small_limit(old)
