"""Fewer spectra than half the SMs against an index of more than 2^16 entries: each is searched
by several CTAs. All of a length's entries, parts of some, none, peaks that repeat, intensities
that need the wide search, spectra of the small-window search between them; all equal the oracle."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu

_CACHE = {}


def _setup():
    if not _CACHE:
        from hicops_gb300 import dslim
        from oracle import oracle as O
        p = S.SearchParams(maxz=3, dF=1, dM=500.0, threads=8, vmods_per_pep=2, mods=[("M", 15.99, 2)])
        db = S.make_database(60000, 5800, p)
        ix = dslim.Index(p)
        ix.construct_all(db)
        _CACHE["x"] = (p, db, ix, O.OracleIndex(db, p))
    return _CACHE["x"]


# up to 32 parts of one spectrum, 8 of 19, two of 76, then one CTA each (152 SMs); twice, as the
# second call finds what the first left in the sums
@pytest.mark.parametrize("nspec", [1, 2, 5, 19, 20, 76, 77])
def test_few_spectra_equal_oracle(nspec):
    p, db, ix, orc = _setup()
    q = S.make_queries(db, nspec, 5810 + nspec, p, peaks=(20, 150),
                       window_mix=[(0.6, "da", 6000.0), (0.2, "da", 900.0), (0.1, "da", 20.0), (0.1, "ppm", 10.0)])
    i = q.idx.astype(np.int64)
    moz, inten, dM = q.moz.copy(), q.intensity.copy(), q.dM.copy()
    dM[0] = 6000.0
    h = (i[1] - i[0]) // 2
    moz[i[0] + h:i[0] + 2 * h] = moz[i[0]:i[0] + h]  # every peak twice
    if nspec > 4:
        dM[1:4] = 6000.0
        inten[i[1]] += 1 << 17   # redone wide
        moz[i[2]:i[3]] = 0       # no valid peak
        dM[4] = -1.0             # no window
    q = S.QueryBatch(idx=q.idx, moz=moz, intensity=inten, precurse=q.precurse, charges=q.charges, rtimes=q.rtimes,
                     dM=dM)
    ores, ohist = orc.query(q, tie_rule=1)
    for _ in range(2):
        compare(*ix.query(q), ores, ohist)


def test_shape_read_and_set_back():
    """Setting back the shape that was read leaves a context as it was: a new one launches what it
    picks (both searches here), a set one what was set."""
    p, db, ix, orc = _setup()
    from hicops_gb300 import dslim
    q = S.make_queries(db, 300, 5899, p)
    ores, ohist = orc.query(q, tie_rule=1)
    new = dslim.Index(p)
    new.construct_all(db)

    def launches():
        compare(*new.query(q), ores, ohist)
        return new.last_launch_count()

    picked, saved = launches(), new.tuning()
    new.set_tuning(**saved)
    assert launches() == picked
    new.set_tuning(tile=4096, threads=512)
    fixed, shape = launches(), new.tuning()
    assert fixed == picked - 1
    new.set_tuning(**shape)
    assert launches() == fixed
    new.set_tuning(**saved)
    assert launches() == picked
    new.close()
