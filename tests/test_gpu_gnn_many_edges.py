"""A training step with more message rows than 65535 chunks of the weight-gradient kernel hold."""
import numpy as np
import pytest

from tessera_b200 import instances, learned

pytestmark = pytest.mark.gpu


def test_gradient_of_many_copies_is_that_of_one():
    """Losses are means over graphs and labelled spins, so copies of one instance leave loss and gradient
    alone: 2100 copies of 4032 directed edges are 66150 chunks of 128 rows.  To 1e-3 in norm: FP32 sums of
    about 10^5 terms each, rounding by 2^-24 sqrt(10^5) = 2e-5 of their magnitudes."""
    rng = np.random.Generator(np.random.PCG64(1))
    ei, ej = np.triu_indices(64, 1)
    p = instances.Problem(rng.uniform(-0.2, 0.2, 64), ei.astype(np.int64), ej.astype(np.int64),
                          rng.uniform(-1, 1, len(ei)) * 0.05)
    net = learned.ScheduleGNN(hidden=8, layers=1, knots=4, seed=3)
    spins = np.where(rng.random(64) < 0.5, 1.0, 0.0).astype(np.float32)

    def step(copies):
        knots = np.tile(np.linspace(0.0, 1.0, 4)[None, :] ** 1.5, (copies, 1))
        return net.train_step([p] * copies, knots, np.tile(spins, copies), lr=0.0, want_grads=True)

    l1, g1 = step(1)
    l2, g2 = step(2100)
    net.close()
    assert l2 == pytest.approx(l1, rel=1e-3)
    assert np.linalg.norm(g2 - g1) < 1e-3 * np.linalg.norm(g1)
