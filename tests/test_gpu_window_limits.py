"""Precursor windows whose limits lie on, just beside and past the entries' masses, in
lengths of one entry to some hundreds, equal masses among them; all equal the oracle."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu


# 216 spectra are searched four ways, 12 times as many in halves
@pytest.mark.parametrize("times", [1, 12])
@pytest.mark.parametrize("npep", [1, 4, 40, 600, 6000])
def test_window_limits_equal_oracle(npep, times):
    from hicops_gb300 import dslim
    from oracle import oracle as O
    p = S.SearchParams(maxz=2, dF=2, dM=500.0, threads=8, vmods_per_pep=2, mods=[("M", 15.99, 2)])
    db = S.make_database(npep, 5500 + npep, p)
    ix = dslim.Index(p)
    ix.construct_all(db)
    mass = np.concatenate([np.asarray(ix.entries(L)["mass"], np.float32) for L in db])
    rng = np.random.default_rng(npep)
    pick = rng.choice(np.unique(mass), 24)
    pick[:2] = mass.min(), mass.max()
    lim = np.concatenate([pick, np.nextafter(pick, np.float32(0)), np.nextafter(pick, np.float32(1e9))])
    # either limit of the window on the mass: precursor = mass + dM, - dM and the mass itself
    dM = rng.choice([0.0, 0.25, 64.0, 500.0, 1e6], 3 * lim.size)
    prec = (np.concatenate([lim, lim, lim]) + dM * np.repeat([0.0, 1.0, -1.0], lim.size)).astype(np.float32)
    prec[-2:] = 0.0, 1e9
    prec, dM = np.tile(prec, times), np.tile(dM, times)
    q = S.make_queries(db, prec.size, 5600, p)
    q = S.QueryBatch(idx=q.idx, moz=q.moz, intensity=q.intensity, precurse=prec, charges=q.charges, rtimes=q.rtimes,
                     dM=dM)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    assert ores["cpsms"].sum() > 0 or npep < 40
    compare(*ix.query(q), ores, ohist)
