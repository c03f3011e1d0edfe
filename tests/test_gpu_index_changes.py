"""Searches after a length of the index was taken out, added or built anew on the same context."""
import numpy as np
import pytest

from tests._util import case

pytestmark = pytest.mark.gpu


def _bytes(r):
    return [np.ascontiguousarray(x).view(np.uint8) for x in r]


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(_bytes(a), _bytes(b)))


def _bad_residue(ix, p, L, seqs):
    s = seqs.copy()
    s[-1, 0] = ord("a")
    ix.construct(L, s)


def _bad_offsets(ix, p, L, seqs):
    e, bA, iA = ix.export(L)
    b = bA.copy()
    b[:-1][b[:-1] == 0] = 1  # descends somewhere, ends as it should
    b[0] = 2
    ix.load(L, seqs, e, b, iA)


def _bad_order(ix, p, L, seqs):
    e = ix.entries(L)
    e["seqid"][0] = seqs.shape[0]
    ix.construct(L, seqs, order=e)


@pytest.mark.parametrize("refused", [_bad_residue, _bad_offsets, _bad_order])
def test_search_after_a_refused_length(refused):
    """A refused call has given the length's arrays up: the search is that of the other lengths."""
    from hicops_gb300 import dslim
    from hicops_gb300._lib import HcError
    p, db, q = case("mods", 5000, 200, 771)
    ix, other = dslim.Index(p), dslim.Index(p)
    ix.construct_all(db)
    ix.query(q)
    with pytest.raises(HcError):
        refused(ix, p, 15, db[15])
    assert ix.info(15) == (0, 0)
    other.construct_all({L: s for L, s in db.items() if L != 15})
    assert _equal(ix.query(q), other.query(q))
    ix.construct(15, db[15])
    other.construct(15, db[15])
    assert _equal(ix.query(q), other.query(q))
    ix.close()
    other.close()


# ---- a captured graph does not outlive what its kernels name ----

def _run(ix, args, d, n, learned=None):
    """Results and histograms (and learned log10 e) of a graph query, or of the plain one."""
    import torch
    from tests.test_gpu_batched_learned import _results
    for t in (d["out"], d["hist"]):
        t.zero_()
    torch.cuda.synchronize()
    if learned is None:
        ix.query_device(*args)
    elif learned is False:
        ix.query_graph(*args)
    else:
        ix.query_learned(learned, *args)
    torch.cuda.synchronize()
    return _results(d, n)


def _added(ix, p, db, q):
    ix.construct(15, db[15])


def _replaced(ix, p, db, q):
    for L in range(p.min_len, p.max_len + 1):
        ix.construct(L, db[L][: db[L].shape[0] // 3])


def _refused(ix, p, db, q):
    from hicops_gb300._lib import HcError
    with pytest.raises(HcError):
        _bad_residue(ix, p, 14, db[14])


def _larger_batch(ix, p, db, q):
    ix.query(q)


def _phase_timing_off(ix, p, db, q):
    ix.set_phase_timing(False)


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("change", [_added, _replaced, _refused, _larger_batch, _phase_timing_off])
def test_graph_after_a_change(change, learned):
    from hicops_gb300 import dslim
    from tests.test_gpu_batched_learned import _dev
    p, db, big = case("mods", 5000, 2000, 781)
    q = big.slice(0, 100)
    ix, fresh = dslim.Index(p), dslim.Index(p)
    nets = [dslim.MLP(x, seed=3) for x in (ix, fresh)] if learned else None
    ix.construct_all({L: s for L, s in db.items() if L != 15})
    d, args = _dev(q)
    if change is _phase_timing_off:
        ix.set_phase_timing(True)
    for _ in range(2):
        _run(ix, args, d, q.nspec, nets[0] if learned else False)
    change(ix, p, db, big)
    got = _run(ix, args, d, q.nspec, nets[0] if learned else False)
    # the same index on a context of its own
    for L in range(p.min_len, p.max_len + 1):
        n, _ = ix.info(L)
        if n:
            fresh.load(L, ix.seqs[L], *ix.export(L))
    exp = _run(fresh, args, d, q.nspec, nets[1] if learned else None)
    assert _equal(got, exp)
    for m in nets or ():
        m.close()
    ix.close()
    fresh.close()


def test_graph_with_another_network():
    """The network of a captured graph is destroyed and others are made, one of which may take its
    place on the host; and the scratch of a network grows."""
    from hicops_gb300 import dslim
    from tests.test_gpu_batched_learned import _dev
    p, db, big = case("mods", 3000, 600, 791)
    q = big.slice(0, 50)
    ix = dslim.Index(p)
    ix.construct_all(db)
    d, args = _dev(q)
    db_, bargs = _dev(big)
    a = dslim.MLP(ix, seed=3)
    exp = _run(ix, args, d, q.nspec, a)
    _run(ix, bargs, db_, big.nspec, a)
    assert _equal(_run(ix, args, d, q.nspec, a), exp)
    w = a.params()
    a.close()
    for _ in range(4):
        m = dslim.MLP(ix, seed=4)
        m.set_params(w)
        assert _equal(_run(ix, args, d, q.nspec, m), exp)
        m.close()
    ix.close()
