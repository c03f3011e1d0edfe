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
