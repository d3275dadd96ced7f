"""The training kernels at the edges of their blocks (64 samples each, tiles of 4 x 4): batches around one block, a
batch of one, many blocks, samples of empty sites. The gradient against the FP64 oracle with the tolerances of the
1024-sample test (one-ulp BF16 differences of hidden activations), and an Adam step against the gradient call."""
import numpy as np
import pytest

from helpers import M
from oracle import learned as L

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def batch(n, seed, empty):
    rng = np.random.default_rng(seed)
    v = np.array([0.3, 0.2, 1.0]) + 0.5 * rng.normal(size=(n, 7, 3))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    f = np.zeros((n, 8), np.float32)
    f[:, :7] = L.features(v[:, 1:], np.ones((n, 6)), 0.6)
    f[:, 7] = 1.0
    d = v[:, 0].astype(np.float32)
    if empty:
        gone = rng.random(n) < 0.3
        gone[0] = False
        f[gone], d[gone] = 0.0, 0.0
    return f, d


@pytest.mark.parametrize("n,empty", [(1, False), (63, True), (64, False), (65, False), (200, True), (4097, True)])
def test_gradient_and_step_at_block_edges(n, empty):
    f, d = batch(n, n, empty)
    rng = np.random.default_rng(1)
    p = L.init_params(3)
    p = (p + 0.3 * rng.normal(size=p.size) * np.abs(p).mean()).astype(np.float32)
    p[-2] += 3.0  # a clear axis bias, so that no sample's axis gradient is ill conditioned
    ft, dt = torch.from_numpy(f).cuda(), torch.from_numpy(d).cuda()
    t = M.Trainer(p, max(n, 64))
    torch.cuda.synchronize()
    loss, g = t.gradient(ft.data_ptr(), dt.data_ptr(), n)
    ok = f[:, 7] != 0
    ref_loss, ref_g = L.loss_and_grad(p.astype(np.float64), f[ok, :7].astype(np.float64), d[ok].astype(np.float64))
    share = ok.sum() / n  # the mean is over the batch, empty rows included
    assert abs(loss - ref_loss * share) < 1e-4 * max(1.0, abs(ref_loss))
    assert np.abs(g - ref_g * share).max() < 5e-3 * np.abs(ref_g).max()
    assert np.linalg.norm(g - ref_g * share) < 1e-2 * np.linalg.norm(ref_g)
    # the step's loss is the gradient's, its update the first Adam step (m / bc1 = g, sqrt(v / bc2) = |g|)
    assert t.step(ft.data_ptr(), dt.data_ptr(), n, 1e-3) == loss
    big = np.abs(g) > 1e-6
    step = t.params().astype(np.float64) - p
    np.testing.assert_allclose(step[big], -1e-3 * np.sign(g[big]), rtol=2e-2, atol=5e-7)
    assert t.gradient(ft.data_ptr(), dt.data_ptr(), n)[0] != loss
    t.close()
