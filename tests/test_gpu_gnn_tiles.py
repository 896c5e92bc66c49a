"""The schedule network's tiled products at the edges of their 32 x 32 tiles and 128-row chunks,
against float64 autograd."""
import numpy as np
import pytest
import torch

from oracle import gnn_oracle
from tessera_b200 import instances, learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,layers,knots", [(8, 1, 2), (31, 2, 16), (33, 2, 32), (64, 3, 16), (72, 1, 7)])
@pytest.mark.parametrize("sizes", [(1,), (1, 2, 5), (30, 35), (12,) * 11])
def test_gradients_match_autograd(monkeypatch, hidden, layers, knots, sizes):
    """FP32 weights and sums of a few hundred terms: 1e-5 relative in the 2-norm leaves a factor of
    ten over sqrt(400) x 6e-8."""
    rng = np.random.Generator(np.random.PCG64(hidden + len(sizes)))
    probs = [instances.dense_er(n, seed=k) if n > 1 else
             instances.Problem(np.array([0.3]), np.zeros(0, np.int64), np.zeros(0, np.int64), np.zeros(0))
             for k, n in enumerate(sizes)]
    net = learned.ScheduleGNN(hidden=hidden, layers=layers, knots=knots, seed=3, bf16=False)
    w = (0.15 * rng.normal(size=net.param_count)).astype(np.float32)
    net.set_params(w)
    tk = np.sort(rng.random((len(sizes), knots)), axis=1)
    ts = (rng.random(sum(sizes)) < 0.5).astype(np.float32)
    _, g = net.train_step(probs, tk, ts, lr=0.0, want_grads=True)
    # The oracle's loss clamps p at 1e-7 and loses the gradient there; the kernels' is the unclamped
    # cross-entropy's, p - t, also where p is 0 or 1 to the last digit.  It is formed from the logits,
    # which the oracle's forward returns with its sigmoid out of the way.
    monkeypatch.setattr(torch, "sigmoid", lambda x: x)
    theta = torch.tensor(w, dtype=torch.float64, requires_grad=True)
    kn, z = gnn_oracle.forward(theta, probs, hidden, layers, knots)
    bce = torch.nn.functional.binary_cross_entropy_with_logits(z, torch.tensor(ts, dtype=torch.float64))
    (((kn - torch.tensor(tk)) ** 2).mean() + 0.2 * bce).backward()
    g_ref = theta.grad.numpy()
    net.close()
    assert np.linalg.norm(g - g_ref) < 1e-5 * np.linalg.norm(g_ref)
