"""Tiled layer products of the learned solver's network at the edges of their tiles (rows around 16,
32, 64 and the switch to large tiles; widths around 16, 32, 64), against the FP64 restatement.

Tolerance: an FP32 sum of K products of values below 1 is off by at most K 2^-24 of the sum of their
magnitudes per layer, 4 layers of at most 130: 3e-5; the gradients' row sums are cut into chunks of
about 1,000 rows at most, 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n_in,hidden,layers,n_out", [
    (1, 1, 1, 1, 1), (15, 31, 33, 1, 5), (17, 16, 15, 2, 32), (64, 65, 64, 3, 63), (65, 87, 64, 3, 108), (255, 22, 32, 0, 30),
    (257, 5, 129, 1, 2), (9727, 87, 64, 1, 108), (9729, 33, 65, 2, 17)])
def test_layers(tpss, cuda, rows, n_in, hidden, layers, n_out):
    import torch
    from oracle import np_mlp
    rng = np.random.Generator(np.random.Philox(rows + n_in))
    m = tpss.MLP(n_in, n_out, hidden, layers)
    params = (rng.uniform(-1, 1, m.n_params) / np.sqrt(max(n_in, hidden))).astype(np.float32)
    m.set_params(params)
    x = rng.uniform(-1, 1, (rows, n_in)).astype(np.float32)
    t = rng.uniform(-1, 1, (rows, n_out)).astype(np.float32)
    widths = [n_in] + [hidden] * layers + [n_out]
    y_ref, _ = np_mlp.forward(params, widths, x)
    loss_ref, g_ref = np_mlp.loss_grad(params, widths, x, t)
    xd, td = torch.tensor(x, device=cuda), torch.tensor(t, device=cuda)
    y = m.forward(xd).cpu().numpy()
    loss, g = m.loss_grad(xd, td)
    assert np.abs(y - y_ref).max() <= 3e-5 * np.abs(y_ref).max()
    assert abs(loss - loss_ref) <= 3e-5 * loss_ref
    assert np.linalg.norm(g - g_ref) <= 1e-4 * np.linalg.norm(g_ref)
    loss2, g2 = m.loss_grad(xd, td)
    assert loss2 == loss and np.array_equal(g, g2)
