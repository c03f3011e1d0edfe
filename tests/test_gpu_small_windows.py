"""The search of small windows and the launch shapes a context picks by itself: batches
below and above the lines of that choice, windows from none to all candidates of a
length, peak lists from none to 100, the widest bins; all equal the oracle."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu

_CACHE = {}


def _setup(npep, dF):
    if (npep, dF) not in _CACHE:
        from hicops_gb300 import dslim
        from oracle import oracle as O
        p = S.SearchParams(maxz=3, dF=dF, dM=500.0, threads=8, vmods_per_pep=2, mods=[("M", 15.99, 2)])
        db = S.make_database(npep, 5200, p)
        ix = dslim.Index(p)
        ix.construct_all(db)
        _CACHE[(npep, dF)] = (p, db, ix, O.OracleIndex(db, p))
    return _CACHE[(npep, dF)]


# 3,000 peptides: every window small; 45,000 (77,000 entries, more than 2^16): windows on
# both sides of 2^15 candidates at 6,000 Da; 152 spectra: one per SM; 1,024: passed over, past
# it: ordered
@pytest.mark.parametrize("npep,dF,nspec", [(3000, 1, 1), (3000, 1, 700), (3000, 16, 40), (45000, 1, 3), (45000, 1, 152),
                                           (45000, 1, 153), (45000, 1, 1024), (45000, 1, 1025)])
def test_picked_shapes_equal_oracle(npep, dF, nspec):
    p, db, ix, orc = _setup(npep, dF)
    q = S.make_queries(db, nspec, 5300 + nspec, p, peaks=(0, 150),
                       window_mix=[(0.3, "ppm", 10.0), (0.2, "da", 20.0), (0.2, "da", 500.0), (0.3, "da", 6000.0)])
    idx, moz = q.idx.astype(np.int64), q.moz.copy()
    if nspec > 2:
        moz[idx[0]:idx[1]] = 0       # no valid peak
        q.dM[1] = -1.0               # no window
        h = (idx[3] - idx[2]) // 2   # every peak twice: counts past one per bucket
        moz[idx[2] + h:idx[2] + 2 * h] = moz[idx[2]:idx[2] + h]
    q = S.QueryBatch(idx=q.idx, moz=moz, intensity=q.intensity, precurse=q.precurse, charges=q.charges,
                     rtimes=q.rtimes, dM=q.dM)
    ores, ohist = orc.query(q, tie_rule=1)
    compare(*ix.query(q), ores, ohist)


def test_small_windows_overflow_goes_wide():
    """Intensities from 2^17 on and more than 63 equal peaks on one class key: redone wide."""
    p, db, ix, orc = _setup(3000, 1)
    q = S.make_queries(db, 30, 5400, p, window_mix=[(1.0, "da", 100.0)])
    inten, moz = q.intensity.copy(), q.moz.copy()
    i = q.idx.astype(np.int64)
    inten[i[0]:i[1]] += 1 << 17
    moz[i[1]:i[2]] = 14711 + np.arange(i[2] - i[1]) % 2  # about y1 of K at charge 1
    q = S.QueryBatch(idx=q.idx, moz=moz, intensity=inten, precurse=q.precurse, charges=q.charges, rtimes=q.rtimes,
                     dM=q.dM)
    ores, ohist = orc.query(q, tie_rule=1)
    res, hist = ix.query(q)
    compare(res, hist, ores, ohist)
    assert res["flags"][0] & 0x100
