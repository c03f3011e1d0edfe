"""Gradients and training steps of the learned tail's network at the sizes where
the tiling changes (rows of a tile, tiles of an SM, a ragged last tile or
minibatch), against the float64 restatement."""
import numpy as np
import pytest

from hicops_gb300 import synthetic as S
from tests.test_gpu_batched_learned import _np_forward_backward

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(-2, 1.5, size=(n, 256)).astype(np.float32)
    Y = np.stack([rng.uniform(-0.5, -0.05, n), rng.uniform(0, 6, n), rng.uniform(0, 80, n),
                  rng.uniform(0, 0.3, n)], 1).astype(np.float32)
    Y[::5, 2:] = np.nan
    return X, Y


@pytest.mark.parametrize("n", [1, 8, 9, 1216, 1217, 2432, 2433, 4864, 4901])
def test_gradients_at_tile_edges(n):
    """FP32 sums of n terms: each share's error is below n/shares * 2^-24 of the sum of
    magnitudes, 2e-4 of the largest gradient at these sizes with a wide margin."""
    import torch
    from hicops_gb300 import dslim
    ix = dslim.Index(S.SearchParams(maxz=2))
    m = dslim.MLP(ix, seed=9)
    X, Y = _data(n, n)
    dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
    g, loss = m.gradients(dX.data_ptr(), dY.data_ptr(), n)
    g2, loss2 = m.gradients(dX.data_ptr(), dY.data_ptr(), n)
    assert np.array_equal(g, g2) and loss == loss2  # a fixed order of every sum
    g64, loss64, _ = _np_forward_backward(m.params().astype(np.float64), X.astype(np.float64), Y.astype(np.float64))
    assert abs(loss - loss64) <= 1e-4 * max(1.0, abs(loss64))
    assert np.abs(g - g64).max() <= 2e-4 * np.abs(g64).max()
    m.close()
    ix.close()


@pytest.mark.parametrize("n,batch", [(250, 100), (1300, 1250)])
def test_training_follows_float64_adam(n, batch):
    """Two epochs with a ragged last minibatch against Adam in float64. Where a
    gradient is smaller than its own rounding (about 1e-4 of the weights) the sign
    of Adam's first step is open, so the path as a whole is compared: within 5 %
    of its length."""
    import torch
    from hicops_gb300 import dslim
    ix = dslim.Index(S.SearchParams(maxz=2))
    m = dslim.MLP(ix, seed=11)
    X, Y = _data(n, n + 1)
    dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
    p0 = m.params().astype(np.float64)
    loss = m.train(dX.data_ptr(), dY.data_ptr(), n, batch=batch, epochs=2, lr=1e-4)
    p, mo, ve, t = p0.copy(), 0.0, 0.0, 0
    for _ in range(2):
        losses = []
        for a in range(0, n, batch):
            g, l64, _ = _np_forward_backward(p, X[a:a + batch].astype(np.float64), Y[a:a + batch].astype(np.float64))
            losses.append(l64)
            t += 1
            mo, ve = 0.9 * mo + 0.1 * g, 0.999 * ve + 0.001 * g * g
            p = p - 1e-4 * (mo / (1 - 0.9 ** t)) / (np.sqrt(ve / (1 - 0.999 ** t)) + 1e-8)
    assert np.linalg.norm(m.params() - p) <= 0.05 * np.linalg.norm(p - p0)
    assert abs(loss - np.mean(losses)) <= 1e-3 * max(1.0, abs(np.mean(losses)))
    m.close()
    ix.close()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2432, 2433, 2465, 4864, 4865, 9728, 9729, 9761, 9791, 10001, 14592,
                               14593])
def test_inference_at_tile_edges(n):
    """Both inference kernels at the edges of their tiles, of the line between them (16
    spectra per SM of a 152-SM part) and of the last wave's half tiles, and nothing written past the last spectrum.
    256 + 128 + 64 FP32 terms: within 448 * 2^-24 of the largest output."""
    import torch
    from hicops_gb300 import dslim
    ix = dslim.Index(S.SearchParams(maxz=2))
    m = dslim.MLP(ix, seed=13)
    X, Y = _data(n, n + 2)
    dX = torch.from_numpy(X).cuda()
    out = torch.full((n * 4 + 65,), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for at in (0, 1):  # the outputs may start at any float
        m.forward(dX.data_ptr(), n, out.data_ptr() + 4 * at)
        torch.cuda.synchronize()
        o = out.cpu().numpy()
        _, _, o64 = _np_forward_backward(m.params().astype(np.float64), X.astype(np.float64), Y.astype(np.float64))
        assert np.abs(o[at:at + 4 * n].reshape(n, 4) - o64).max() <= 448 * 2.0 ** -24 * np.abs(o64).max()
        assert (o[at + 4 * n:] == 7.0).all()
    m.close()
    ix.close()


def test_gradients_of_inputs_at_any_float():
    """Inputs that start 4 bytes past a 16-byte boundary give the same gradients."""
    import torch
    from hicops_gb300 import dslim
    ix = dslim.Index(S.SearchParams(maxz=2))
    m = dslim.MLP(ix, seed=9)
    X, Y = _data(70, 1)
    dY = torch.from_numpy(Y).cuda()
    buf = torch.zeros(70 * 256 + 4, dtype=torch.float32, device="cuda")
    g = []
    for at in (0, 1):
        buf[at:at + 70 * 256] = torch.from_numpy(X).reshape(-1).cuda()
        torch.cuda.synchronize()
        g.append(m.gradients(buf.data_ptr() + 4 * at, dY.data_ptr(), 70)[0])
    assert np.array_equal(g[0], g[1])
    m.close()
    ix.close()
