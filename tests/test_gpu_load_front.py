"""A loaded index whose bucket offsets do not start at 0: the postings in front of the first
bucket lie in none and are not searched, and the offsets stay as they were given."""
import os

import numpy as np
import pytest

from hicops_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upto", [1, 4500, 6500, 100000, None])
def test_postings_in_front_of_the_first_bucket(upto, tmp_path):
    """The postings of the buckets below `upto` (all of them: None) in front. Below bucket 7000
    lie b ions of one residue (at most 70 m/z; the lightest y ion is K's at 74): the search is then
    that of an index with those postings in bucket 0, which no peak reaches."""
    from hicops_gb300 import dslim
    p = S.SearchParams(min_len=9, max_len=9, maxz=2, dF=1, dM=300.0, threads=4)
    db = S.make_database(3000, 91, p)
    q = S.make_queries(db, 60, 92, p)
    # peaks on every bucket in question too: noise starts at 100 m/z
    moz = q.moz.copy()
    i = q.idx.astype(np.int64)
    for s in range(0, 60, 2):
        moz[i[s]:i[s] + 10] = np.linspace(3000, 6900, 10).astype(np.uint32)
    q = S.QueryBatch(idx=q.idx, moz=moz, intensity=q.intensity, precurse=q.precurse, charges=q.charges,
                     rtimes=q.rtimes)
    a, b, c, d = (dslim.Index(p) for _ in range(4))
    a.construct_all(db)
    e, bA, iA = a.export(9)
    k = int(bA[-1 if upto is None else upto])
    front = np.maximum(bA, np.uint32(k))
    b.load(9, db[9], e, front, iA)
    rb, hb = b.query(q)
    if upto is not None and upto <= 7000:
        bA0, iA0 = front.copy(), iA.copy()
        bA0[0] = 0
        iA0[:bA0[1]].sort()  # ids ascend in a bucket
        c.load(9, db[9], e, bA0, iA0)
        rc, hc = c.query(q)
        assert np.array_equal(rb.view(np.uint8), rc.view(np.uint8)) and np.array_equal(hb, hc)
    if upto == 6500:  # (they would have been visited)
        assert k > 0 and (rb["post_bytes"] < a.query(q)[0]["post_bytes"]).any()
    path = os.path.join(tmp_path, "ix.hcd")
    b.save(path)
    d.restore(path)
    for x in (b, d):
        e2, bA2, iA2 = x.export(9)
        assert np.array_equal(e2, e) and np.array_equal(bA2, front)
        assert np.array_equal(iA2[k:], iA[k:]) and not iA2[:k].any()
    rd, hd = d.query(q)
    assert np.array_equal(rb.view(np.uint8), rd.view(np.uint8)) and np.array_equal(hb, hd)
    for x in (a, b, c, d):
        x.close()
