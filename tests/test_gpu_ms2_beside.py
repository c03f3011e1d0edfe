"""hc_ms2_open beside other work: a search left running on a stream does not hold it up."""
import ctypes as C

import numpy as np
import pytest

from oracle import ms2 as M
from hicops_gb300 import synthetic as S
from tests.test_gpu_ms2 import _same
from tests.test_gpu_ms2_device_parse import FORMS, _body

pytestmark = pytest.mark.gpu

HC_ERR_TIMEOUT = -3021
PICK = (100, 100000, 1000)


def _file(tmp_path):
    path = str(tmp_path / "b.ms2")
    text = "".join(_body(np.random.default_rng(5), 300, "\n", FORMS["plain"]))
    assert len(text) > 1 << 16  # the device parser takes it
    open(path, "w").write(text)
    st, o = M.read_ms2(path, *PICK)
    assert st == 0
    return path, o


def _batch(r):
    b, left = r.extractbatch(r.getQAcount())
    assert left == 0
    return dict(idx=b.idx, moz=b.moz, intensity=b.intensity, precurse=b.precurse, charges=b.charges, rtimes=b.rtimes)


@pytest.mark.parametrize("form", ["device", "graph", "noalloc"])
@pytest.mark.parametrize("own", [True, False])
def test_open_while_a_search_runs(own, form, tmp_path):
    """Searches of some hundred milliseconds, on the context's stream or another; they still run when
    the file is open, and the batch is the file's."""
    import torch
    from hicops_gb300 import dslim
    from tests.test_gpu_batched_learned import _dev
    path, o = _file(tmp_path)
    p = S.SearchParams(maxz=3, dF=1, dM=6000.0, threads=8, vmods_per_pep=2, mods=[("M", 15.99, 2)])
    p.base_int, p.min_int = PICK[1], PICK[2]
    db = S.make_database(60000, 5900, p)
    ix = dslim.Index(p)
    ix.construct_all(db)
    q = S.make_queries(db, 4000, 5901, p)
    d, args = _dev(q)
    s = None if own else torch.cuda.Stream()
    handle = None if own else s.cuda_stream

    def search():
        if form == "noalloc":
            ix._check(ix.lib.hc_dslim_query_noalloc(ix.ctx, *[None if x is None else C.c_void_p(x) for x in args[:5]],
                                                    args[5], args[6], C.c_void_p(args[7]), C.c_void_p(args[8]),
                                                    None if own else C.c_void_p(handle)), "noalloc")
        else:
            (ix.query_device if form == "device" else ix.query_graph)(*args, stream=handle)

    torch.cuda.synchronize()
    search()
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    search()
    torch.cuda.synchronize()
    b.record()
    b.synchronize()
    one = a.elapsed_time(b)
    for _ in range(int(400 / one) + 1):
        search()
    r = dslim.MSQuery(ix).initialize(path)
    assert ix.lib.hc_ctx_wait(ix.ctx, None if own else C.c_void_p(handle), 0.0) == HC_ERR_TIMEOUT
    torch.cuda.synchronize()
    _same(_batch(r), o)
    r.DeinitQueryFile()
    ix.close()


def test_read_while_a_graph_is_captured(tmp_path):
    """Opening a file, taking its raw and picked peaks and closing it, inside a capture that forbids
    unsafe calls: the capture ends well, its graph replays, and the file's values are right."""
    import torch
    from hicops_gb300 import _lib as L
    from hicops_gb300 import dslim
    path, o = _file(tmp_path)
    p = S.SearchParams(maxz=2, dF=2, dM=100.0)
    p.base_int, p.min_int = PICK[1], PICK[2]
    ix = dslim.Index(p)
    raw = dslim.read_ms2_raw(path, p.scale)
    off, mz, it = np.zeros_like(raw["off"]), np.zeros_like(raw["mz"]), np.zeros_like(raw["mz"])
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="global"):
        y = x + 1
        r = dslim.MSQuery(ix).initialize(path)
        assert ix.lib.hc_ms2_raw(r.h, 0, r.QAcount, L.ptr(off), L.ptr(mz), L.ptr(it), None, None, None) == 0
        other = dslim.MSQuery(ix).initialize(path)
        within = _batch(other)
        other.DeinitQueryFile()
        z = y * 3
    g.replay()
    torch.cuda.synchronize()
    assert (z == 6).all()
    assert np.array_equal(off, raw["off"]) and np.array_equal(mz, raw["mz"]) and np.array_equal(it, raw["intensity"])
    _same(within, o)
    _same(_batch(r), o)
    r.DeinitQueryFile()
    ix.close()


def test_reader_outlives_its_context(tmp_path):
    """A file's raw peaks are its own: read and closed after the context that parsed it is gone, and
    extracted by another context of the device."""
    from hicops_gb300 import _lib as L
    from hicops_gb300 import dslim
    path, o = _file(tmp_path)
    p = S.SearchParams(maxz=2, dF=2, dM=100.0)
    p.base_int, p.min_int = PICK[1], PICK[2]
    a, b = dslim.Index(p), dslim.Index(p)
    raw = dslim.read_ms2_raw(path, p.scale)
    r = dslim.MSQuery(a).initialize(path)
    a.close()
    off, mz, it = np.zeros_like(raw["off"]), np.zeros_like(raw["mz"]), np.zeros_like(raw["mz"])
    assert a.lib.hc_ms2_raw(r.h, 0, r.QAcount, L.ptr(off), L.ptr(mz), L.ptr(it), None, None, None) == 0
    assert np.array_equal(off, raw["off"]) and np.array_equal(mz, raw["mz"]) and np.array_equal(it, raw["intensity"])
    r.ix = b
    _same(_batch(r), o)
    r.DeinitQueryFile()
    b.close()
