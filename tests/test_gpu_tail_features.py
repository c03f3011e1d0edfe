"""The learned tail's features where the top hit's bin meets the groups of 32 and
128 bins, the fold at bin 255 and the histogram's end, against a float64 restatement."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def test_features_at_every_top_hit_edge():
    import torch
    from hicops_gb300 import dslim
    from hicops_gb300._lib import HC_HIST_BINS, RESULT_DTYPE
    tops = np.array([0, 1, 2, 31, 32, 33, 127, 128, 129, 254, 255, 256, 257, 600, 1001])
    rng = np.random.default_rng(5)
    n = tops.size
    hist = np.zeros((n, HC_HIST_BINS), np.uint32)
    for i, t in enumerate(tops):
        hist[i, :t] = rng.integers(0, 50, t)
        hist[i, t] = 1 + i
    res = np.zeros(n, RESULT_DTYPE)
    res["cpsms"] = hist.sum(1)
    res["hyperscore"] = tops.astype(np.float32) / np.float32(10)
    ix = dslim.Index(S.SearchParams(maxz=2))
    m = dslim.MLP(ix)
    dh = torch.from_numpy(hist.view(np.int32)).cuda()
    dr = torch.from_numpy(res.view(np.uint8)).cuda()
    x = torch.full((n + 1, 256), 9.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    m.features(dh.data_ptr(), dr.data_ptr(), n, x.data_ptr())
    torch.cuda.synchronize()
    got = x.cpu().numpy()
    h = hist[:, :256].astype(np.float64)
    h[:, 255] += hist[:, 256:].sum(1)
    c = hist.sum(1).astype(np.float64)[:, None]
    want = np.log10(np.maximum((c - h.cumsum(1)) / c, 1e-7))
    for i, t in enumerate(np.minimum(tops, 256)):
        want[i, t:] = want[i, t - 1] if t else 0.0
    # a float quotient (2 roundings) and log10f (2 ulp of values up to 7)
    assert np.abs(got[:n] - want).max() <= 2e-6
    assert (got[n] == 9.0).all()
    m.close()
    ix.close()
