"""The scorecard's start between two jobs of a spectrum: peaks at the y1 keys of no entry
class, of one and of two, in windows of whole and of ragged tiles; all equal the oracle."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,ctas", [(128, 1), (512, 2), (1024, 1)])
def test_classes_matched_equal_oracle(threads, ctas):
    from hicops_gb300 import dslim
    from oracle import oracle as O
    p = S.SearchParams(maxz=3, dF=1, dM=500.0, threads=8, vmods_per_pep=2, mods=[("M", 15.99, 2)])
    db = S.make_database(60000, 5700, p)
    ix = dslim.Index(p)
    ix.construct_all(db)
    ix.set_tuning(threads=threads, ctas_per_sm=ctas, tile=2048, schedule=0)
    q = S.make_queries(db, 24, 5701, p, peaks=(60, 90),
                       window_mix=[(0.5, "da", 6000.0), (0.3, "da", 300.0), (0.2, "da", 20.0)])
    moz, i = q.moz.copy(), q.idx.astype(np.int64)
    k1, r1 = 14711, 17511  # y1 of K and of R at charge 1
    low = moz < 18000
    moz[low] += 18000  # no peak near a y1 key
    for s in range(q.nspec):
        if s % 4 & 1:
            moz[i[s]] = k1 + s % 3 - 1
        if s % 4 & 2:
            moz[i[s] + 1] = r1
    q = S.QueryBatch(idx=q.idx, moz=moz, intensity=q.intensity, precurse=q.precurse, charges=q.charges,
                     rtimes=q.rtimes, dM=q.dM)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    assert ores["cpsms"].sum() > 0
    compare(*ix.query(q), ores, ohist)
    ix.close()
