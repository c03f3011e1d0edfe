"""Peaks that repeat one key so often that a candidate's shared-ion count of one series comes to
127, 128 and past it: from 128 on the packed words do not hold and the spectrum is redone wide.
In the general search, the small-window search and with a spectrum in parts."""
import numpy as np
import pytest

from hicops_gb300 import _lib as HL
from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npep,nspec,shape", [(2000, 40, None), (2000, 40, dict(tile=2048, threads=256)),
                                              (60000, 12, None)])
@pytest.mark.parametrize("times", [31, 32, 42, 43, 63, 64, 65, 100])
def test_counts_about_128(times, npep, nspec, shape):
    from hicops_gb300 import dslim
    from oracle import oracle as O
    # wide bins: a candidate has one to four ions of a series at a key
    p = S.SearchParams(min_len=18, max_len=22, maxz=2, dF=16, dM=3000.0, threads=8, scale=20, min_cpsm=1)
    db = S.make_database(npep, 601, p)
    q = S.make_queries(db, nspec, 602, p)
    idx, moz, inten = [0], [], []
    rng = np.random.default_rng(times)
    for s in range(nspec):
        a, b = int(q.idx[s]), int(q.idx[s + 1])
        key = int(np.median(q.moz[a:b])) + int(rng.integers(-400, 400))
        moz.append(np.full(times, key, np.uint32))
        inten.append(np.sort(rng.integers(1000, 100001, times)).astype(np.uint32))
        idx.append(idx[-1] + times)
    q = S.QueryBatch(idx=np.array(idx, np.uint32), moz=np.concatenate(moz), intensity=np.concatenate(inten),
                     precurse=q.precurse, charges=q.charges, rtimes=q.rtimes)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    ix = dslim.Index(p)
    ix.construct_all(db)
    if shape:
        ix.set_tuning(**shape)
    res, hist = ix.query(q)
    compare(res, hist, ores, ohist, fit_exact_min=0.0)
    if times == 64:  # twice 64 among them
        assert (ores["sharedions"] >= 128).any() and (res["flags"] & HL.FLAG_WIDE).any()
    ix.close()
