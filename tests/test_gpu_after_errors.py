"""A call that fails leaves nothing behind that makes the next one fail."""
import ctypes as C

import numpy as np
import pytest

from tests._util import case

pytestmark = pytest.mark.gpu


def _no_rows(ix):
    from hicops_gb300 import dslim
    from hicops_gb300._lib import HcError
    import torch
    m = dslim.MLP(ix, seed=1)
    x = torch.zeros(256, device="cuda")
    with pytest.raises(HcError):
        m.gradients(x.data_ptr(), x.data_ptr(), 0)
    m.close()


def _still_running(ix):
    import torch
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(200_000_000)  # ~0.1 s
    assert ix.lib.hc_ctx_wait(ix.ctx, C.c_void_p(s.cuda_stream), 0.001) == -3021


@pytest.mark.parametrize("fails", [_no_rows, _still_running])
def test_search_and_build_after_a_failed_call(fails):
    from hicops_gb300 import dslim
    p, db, q = case("mods", 2000, 50, 731)
    ix = dslim.Index(p)
    ix.construct_all(db)
    r, h = ix.query(q)
    fails(ix)
    r2, h2 = ix.query(q)
    assert np.array_equal(r.view(np.uint8), r2.view(np.uint8)) and np.array_equal(h, h2)
    fails(ix)
    ix.construct(20, db[20])
    r2, h2 = ix.query(q)
    assert np.array_equal(r.view(np.uint8), r2.view(np.uint8)) and np.array_equal(h, h2)
    ix.close()
