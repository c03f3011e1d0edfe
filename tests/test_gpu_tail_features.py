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


def _targets64(h, hyp, cps):
    """Slope and first bin of expeRT's window on the float64 curve, or None."""
    b = np.nonzero(h[:hyp])[0]
    if not b.size:
        return None
    first, last = int(b[0]), int(b[-1])
    last += first == last
    if last - first + 1 < 4:
        return None
    y = np.log10(np.maximum((cps - h.cumsum()[first:last + 1]) / cps, 1e-9))
    t1, t2 = y[0] + 0.22 * (y[-1] - y[0]), y[0] + 0.87 * (y[-1] - y[0])
    low, m2 = np.nonzero(y <= t1)[0], int(np.nonzero(y >= t2)[0][-1])
    mark = min(int(low[0]) - 1, m2 - 1) if low.size else -1
    if mark < 0:
        return None
    return np.polyfit(np.arange(mark, m2 + 1), y[mark:m2 + 1], 1)[0], first + mark


def test_targets_where_the_top_hit_meets_a_lane():
    """The curve where the top hit's and the first bin meet a lane's four bins, the 128 of a
    step and the histogram's end, with histograms that start at any word. Each point of the
    FP32 curve is within 1e-6 (a quotient's rounding and log10f's 2 ulp below 7), and over
    a window of m >= 2 points the slope within 12 / m of that; the first bin is equal."""
    import torch
    from hicops_gb300 import dslim
    from hicops_gb300._lib import HC_HIST_BINS, RESULT_DTYPE
    tops = np.array([0, 1, 3, 4, 5, 6, 7, 8, 9, 60, 126, 127, 128, 129, 130, 131, 132, 133, 255, 256, 257, 600, 999, 1000,
                     1001])
    starts = [0, 1, 2, 3, 5, 127, 128, 129]
    rows = [(t, f) for t in tops for f in starts if f <= t]
    rng = np.random.default_rng(6)
    n = len(rows)
    hist = np.zeros((n, HC_HIST_BINS), np.uint32)
    for i, (t, f) in enumerate(rows):
        k = np.arange(t - f)
        hist[i, f:t] = np.maximum(0, 2e5 * np.exp(-k * rng.uniform(4, 9) / max(t - f, 1)) + rng.integers(0, 3, t - f))
        hist[i, t] = 1
    res = np.zeros(n, RESULT_DTYPE)
    res["cpsms"] = hist.sum(1)
    res["hyperscore"] = np.array([t for t, _ in rows], np.float32) / np.float32(10)
    ix = dslim.Index(S.SearchParams(maxz=2, min_cpsm=1))
    m = dslim.MLP(ix)
    buf = torch.zeros(hist.size + 1, dtype=torch.int32, device="cuda")
    dr = torch.from_numpy(res.view(np.uint8)).cuda()
    got = []
    for at in (0, 1):
        buf[at:at + hist.size] = torch.from_numpy(hist.view(np.int32)).reshape(-1).cuda()
        y = torch.zeros(n, 4, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        m.targets(buf.data_ptr() + 4 * at, dr.data_ptr(), n, y.data_ptr())
        torch.cuda.synchronize()
        got.append(y.cpu().numpy())
    assert np.array_equal(got[0], got[1], equal_nan=True)
    found = 0
    for i, (t, _) in enumerate(rows):
        want = _targets64(hist[i].astype(np.float64), t, float(res["cpsms"][i]))
        if np.isnan(got[0][i, 0]):
            continue  # no window, or a level too near a point
        found += 1
        assert want is not None and got[0][i, 2] == want[1]
        assert abs(got[0][i, 0] - want[0]) <= 12e-6
    assert found >= n // 2
    m.close()
    ix.close()
