"""k_tailfit against the plain form (every step in the reference's order of operations), bit for
bit: histograms as searches leave them, and histograms made so that a point lies on a level of the
regression window or a line's value next to the integer that it is truncated to."""
import ctypes as C

import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from hicops_gb300._lib import HC_HIST_BINS, RESULT_DTYPE

pytestmark = pytest.mark.gpu


def _same_fits(hist, cpsms, top):
    """hist: device int32 [n, bins] with the top hit in; both forms on the same results."""
    import torch
    from hicops_gb300 import dslim
    n = cpsms.size
    res = np.zeros(n, RESULT_DTYPE)
    res["cpsms"] = cpsms
    res["hyperscore"] = (top / 10.0).astype(np.float32)
    ix = dslim.Index(S.SearchParams(min_cpsm=2))
    got = []
    for plain in (0, 1):
        d = torch.from_numpy(res.view(np.uint8).copy()).cuda()
        first = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = ix.lib.hc_check_tailfit(ix.ctx, C.c_void_p(hist.data_ptr()), C.c_void_p(d.data_ptr()), n, plain,
                                     C.c_void_p(first.data_ptr()))
        assert rc == 0
        got.append((np.frombuffer(d.cpu().numpy().tobytes(), RESULT_DTYPE), first.cpu().numpy()))
    ix.close()
    (a, fa), (b, fb) = got
    for f in RESULT_DTYPE.names:
        x, y = (np.ascontiguousarray(v[f]).view(np.uint8).reshape(n, -1) for v in (a, b))
        bad = np.nonzero((x != y).any(1))[0]
        assert bad.size == 0, (f, bad.size, bad[:5], a[f][bad[:5]], b[f][bad[:5]])
    assert np.array_equal(fa, fb)
    return b


def _from_points(first, cum, cps):
    """Device histograms of the curves with cumulative counts cum[n, k] (ascending, the first not
    0) at the bins from first[n] on; what is left of cps lies at the top hit, past the last point."""
    import torch
    n, k = cum.shape
    cnt = np.diff(cum, axis=1, prepend=0)
    assert (cnt >= 0).all() and (cnt[:, 0] > 0).all() and (cum[:, -1] < cps).all()
    top = np.minimum(first + k + 3, HC_HIST_BINS - 1)
    assert (top >= first + k).all()
    h = torch.zeros(n, HC_HIST_BINS, dtype=torch.int64, device="cuda")
    rows = torch.arange(n, device="cuda")
    f, c = torch.from_numpy(first).cuda(), torch.from_numpy(cnt).cuda()
    for j in range(k):
        h[rows, f + j] = c[:, j]
    h[rows, torch.from_numpy(top).cuda()] = torch.from_numpy(cps - cum[:, -1]).cuda()
    return h.to(torch.int32), top


@pytest.mark.parametrize("seed", range(4))
def test_random_histograms(seed):
    """100,000 each: exponential tails of 30 to 10^9 candidates with gaps, steep to flat, from any bin."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(900 + seed)
    n = 100000
    r = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)
    total = 10.0 ** (1.5 + 7.5 * r(n, 1) ** (1 + seed))
    first = (r(n, 1) ** (1 + seed) * 900).floor()
    slope = 10.0 ** (-2.0 + 2.5 * r(n, 1))
    gap = 0.7 * r(n, 1) ** 2
    hist = torch.empty(n, HC_HIST_BINS, dtype=torch.int32, device="cuda")
    bins = torch.arange(HC_HIST_BINS, device="cuda", dtype=torch.float64)[None, :]
    for a in range(0, n, 10000):
        s = slice(a, a + 10000)
        past = (bins - first[s]).clamp(min=0)  # (in front of the first bin the power would overflow)
        x = total[s] * torch.clamp(slope[s], max=1.0) * torch.exp(-slope[s] * past) * (bins >= first[s])
        x = (x + r(*x.shape) * (x > 0.02)) * (r(*x.shape) > gap[s])
        hist[s] = x.floor().clamp(max=5e8).to(torch.int32)
    last = torch.where(hist > 0, bins.to(torch.int32), 0).amax(1)
    top = (last + 1 + (r(n) ** 2 * 40).to(torch.int32)).clamp(max=HC_HIST_BINS - 1)
    hist[torch.arange(n, device="cuda"), top.long()] += 1
    cps = hist.sum(1, dtype=torch.int64).cpu().numpy()
    assert cps.max() < 2 ** 31 and (hist >= 0).all()
    b = _same_fits(hist, cps.astype(np.uint32), top.cpu().numpy())
    assert (b["mu"] != 0).mean() > 0.5


def test_lines_next_to_an_integer():
    """Two-point curves, whose line is known: those of 2 x 10^7 whose slope x 10^6 lies within 10^-6 of
    an integer or whose intercept does within 3 x 10^-5, half of them at the last bins, where a slope's
    last bits move the intercept most."""
    rng = np.random.default_rng(31)
    first, cum, cps, near = [], [], [], [0, 0]
    for _ in range(20):
        n = 1000000
        f = np.where(rng.random(n) < 0.5, rng.integers(980, 996, n), rng.integers(1, 996, n))
        t = np.floor(10.0 ** rng.uniform(2, 9, n)).astype(np.int64)
        c0 = 1 + np.floor(t * rng.random(n) ** 3 * 0.9).astype(np.int64)
        c1 = np.minimum(c0 + 1 + np.floor((t - c0) * rng.random(n)).astype(np.int64), t - 1)
        ok = (c0 < t - 1) & (c1 > c0)
        y0, y1 = (np.log10(1.0 - c / t) for c in (np.minimum(c0, t - 1), np.minimum(c1, t - 1)))
        mu = (y1 - y0) * 1e6
        beta = ((y0 + y1) / 2 - (y1 - y0) * (f + 0.5)) * 1e6
        a = ok & (np.abs(mu - np.rint(mu)) < 1e-6)
        b = ok & (np.abs(beta - np.rint(beta)) < 3e-5)
        near[0] += int(a.sum())
        near[1] += int(b.sum())
        k = a | b
        first.append(f[k])
        cum.append(np.stack([c0, c1], 1)[k])
        cps.append(t[k])
    assert min(near) > 20
    first, cum, cps = (np.concatenate(x) for x in (first, cum, cps))
    hist, top = _from_points(first, cum, cps)
    _same_fits(hist, cps.astype(np.uint32), top)


@pytest.mark.parametrize("level", [0.22, 0.87])
def test_points_on_a_level(level):
    """Curves of seven points with an inner one at the nearest count to a level of the window, and
    one count to either side: within 10^-9 of it (counts up to 2 x 10^9) to within 10^-4 (some 10^3)."""
    rng = np.random.default_rng(int(100 * level))
    n, k = 60000, 7
    t = np.floor(10.0 ** rng.uniform(3, 9.3, n)).astype(np.int64)
    s0, s1 = rng.uniform(0.6, 0.999, n), rng.uniform(0.3, 0.55, n)
    p = rng.integers(1, k - 1, n)
    at = 10.0 ** (np.log10(s0) + level * (np.log10(s1) - np.log10(s0)))
    s = np.where(np.arange(k)[None, :] < p[:, None],
                 s0[:, None] + (at - s0)[:, None] * np.arange(k)[None, :] / p[:, None],
                 at[:, None] + (s1 - at)[:, None] * (np.arange(k)[None, :] - p[:, None]) / (k - 1 - p)[:, None])
    cum = np.rint((1.0 - s) * t[:, None]).astype(np.int64)
    c0, c1 = cum[:, 0].clip(1), cum[:, -1]
    # the level of the curve as it is, and the count nearest to it
    y0, y1 = (np.log10(1.0 - c / t) for c in (c0, c1))
    mid = np.rint((1.0 - 10.0 ** (y0 + level * (y1 - y0))) * t).astype(np.int64)
    cum[np.arange(n), p] = mid + np.arange(n) % 3 - 1
    cum[:, 0] = c0
    ok = (np.diff(cum, axis=1) >= 0).all(1) & (cum[:, -1] < t)
    assert ok.mean() > 0.9
    near = np.abs(np.log10(1.0 - cum[np.arange(n), p] / t) - (y0 + level * (y1 - y0)))
    assert (near[ok] < 1e-9).sum() > 1000 and (near[ok] < 5e-5).mean() > 0.5
    hist, top = _from_points(rng.integers(1, 900, n)[ok], cum[ok], t[ok])
    _same_fits(hist, t[ok].astype(np.uint32), top)
