"""The bucket scans of an index build where they take another level: 4096 tiles of 4096 words are
added up by the last launch, more are scanned themselves. Fine m/z scales make that many buckets."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu

EDGE = 4096 * 4096  # words; a bucket array has max_mass * scale + 1


@pytest.mark.parametrize("max_mass,scale", [(4097, 4095), (4915, 3414), (4999, 3400)])
def test_build_and_search_at_scan_levels(max_mass, scale):
    from hicops_gb300 import dslim
    from oracle import oracle as O
    assert (max_mass * scale + 1 <= EDGE) == (scale == 4095)
    p = S.SearchParams(min_len=12, max_len=12, maxz=2, dF=2, dM=200.0, threads=8, max_mass=max_mass, scale=scale)
    db = S.make_database(2000, 311, p)
    q = S.make_queries(db, 30, 312, p)
    ix = dslim.Index(p)
    ix.construct_all(db)
    e, bA, iA = ix.export(12)
    obA, oiA = O.build_index(db[12], 12, e, p)
    assert np.array_equal(bA, obA) and np.array_equal(iA, oiA)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    compare(*ix.query(q), ores, ohist, fit_exact_min=0.9)
    ix.close()
