"""The first steps of a batch whose cap calls for the LQ: theta of 2 to a few dozen rows, square, wide and tall,
on both sides of the size up to which the batched LQ lets them be."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chi", [(12, 64), (13, 64), (14, 128)])
@pytest.mark.parametrize("steps", [2, 3, 4])
def test_batch_follows_the_single_anneals(n, chi, steps):
    """chi is 2^(n / 2), nothing truncates, so both are the exact evolution up to rounding: 1e-10 after at most 4 steps of 126
    updates at 1e-13 each."""
    probs = [instances.chain_range(n=n, dmax=3, seed=s, T=0.1 * steps, dt=0.1, chi=chi, hzero=False)
             for s in range(3)]
    for p, r in zip(probs, ffi.anneal_batch(probs, chi=chi)):
        o = ffi.anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi, jacobi_precondition=2)
        assert r.max_trunc < 1e-20 and o.max_trunc < 1e-20
        assert abs(r.expected_energy - o.expected_energy) < 1e-10 * max(1.0, abs(o.expected_energy))
        assert np.max(np.abs(r.entropy - o.entropy)) < 1e-10
        assert np.max(np.abs(r.z_expect - o.z_expect)) < 1e-10
        assert abs(r.norm2 - 1.0) < 1e-10
