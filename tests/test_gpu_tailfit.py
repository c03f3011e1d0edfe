"""The tail fit where its short arithmetic meets its edges: spectra with a handful
of candidates (two-point windows, flat curves, a top hit right after the only
other bin), windows that start before the curve, and long curves, against the
oracle's restatement of expeRT."""
import pytest

from tests._util import case, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dM,min_shp,min_cpsm", [(0.01, 1, 1), (0.05, 2, 1), (1.0, 3, 2), (20.0, 4, 4), (500.0, 2, 4)])
def test_tailfit_parity(dM, min_shp, min_cpsm):
    """Every integer of a result equal and the lines of at least 99 % of the spectra; where
    host and device logarithms differ in their last bit a line's slope may truncate one
    millionth away, which moves log10 e by at most 1e-6 x the top hit's bin (< 100 here)."""
    from hicops_gb300 import dslim
    from oracle import oracle as O
    p, db, q = case("mods", 3000, 1500, 4100 + int(10 * dM), dM=dM, min_shp=min_shp, min_cpsm=min_cpsm)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    ix = dslim.Index(p)
    ix.construct_all(db)
    st = compare(*ix.query(q), ores, ohist)
    assert st["reported"] > 0 and st["dlog10e_max"] <= 1e-4
    ix.close()
