"""The index build where its flat kernels have edges: no postings at all, fewer
than a word of 32, whole words, one past them; built, loaded from the reference's
arrays and restored from a file."""
import os

import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests._util import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npep", [0, 1, 2, 31, 32, 33, 700])
def test_build_load_restore_at_word_edges(npep, tmp_path):
    """Length 9 at two charges gives 32 postings an entry (whole words); length 10 36."""
    from hicops_gb300 import dslim
    from oracle import oracle as O
    p = S.SearchParams(min_len=9, max_len=10, maxz=2, dF=1, dM=300.0, threads=4)
    db = S.make_database(1500, 77, p)
    db = {L: db[L][:npep] for L in (9, 10)}
    a, b, c = dslim.Index(p), dslim.Index(p), dslim.Index(p)
    a.construct_all(db)
    for L in (9, 10):
        e, bA, iA = a.export(L)
        obA, oiA = O.build_index(db[L], L, e, p)
        assert np.array_equal(bA, obA) and np.array_equal(iA, oiA)
        b.load(L, db[L], e, bA, iA)
    path = os.path.join(tmp_path, "ix.hcd")
    a.save(path)
    c.restore(path)
    for L in (9, 10):
        for x in (b, c):
            for u, v in zip(a.export(L), x.export(L)):
                assert np.array_equal(u, v)
    src = {L: v for L, v in S.make_database(1500, 77, p).items()}
    q = S.make_queries(src, 40, 78, p)
    ores, ohist = O.OracleIndex(db, p).query(q, tie_rule=1)
    for x in (a, b, c):
        compare(*x.query(q), ores, ohist)
        x.close()


@pytest.mark.parametrize("npep", [2, 3, 1024, 1025, 8191, 8192, 8193, 16400, 19455, 19456, 19457])
def test_entry_order_at_sort_edges(npep):
    """The entries' order where the mass sort changes (one CTA up to 8192 entries, digit
    passes past it; 16 postings an entry, tiles of 2048 of them up to 152 tiles, of 8192
    past that): ascending, equal masses (the sequences have
    four residues, so most masses repeat) in file order; and the postings sorted from them."""
    from hicops_gb300 import dslim
    from oracle import oracle as O
    p = S.SearchParams(min_len=9, max_len=9, maxz=1, dF=1, dM=300.0, threads=8)
    rng = np.random.default_rng(npep)
    seqs = rng.choice(np.frombuffer(b"AGLK", np.uint8), size=(npep, 9))
    ix = dslim.Index(p)
    ix.construct(9, seqs)
    e, bA, iA = ix.export(9)
    mass = S.pep_mass_f32(seqs)
    order = np.argsort(mass, kind="stable")
    assert np.array_equal(e["seqid"], order) and np.array_equal(e["mass"], mass[order])
    obA, oiA = O.build_index(seqs, 9, e, p)
    assert np.array_equal(bA, obA) and np.array_equal(iA, oiA)
    ix.close()
