"""The norm of an anneal that never truncates, with the LQ in front of its Jacobi."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chi,batch", [(10, 32, False), (12, 64, False), (12, 64, True)])
def test_norm_drift_with_the_lq(n, chi, batch):
    """Leftover inner products are proportional to the tolerance and so is the drift of <psi|psi> from 1 (a
    fifth of it at 2e-14 of what 1e-13 leaves): under half of the drift at jacobi_tol = 1e-13, over 12 seeds."""
    probs = [instances.chain_range(n=n, dmax=1, seed=s, T=6.0, dt=0.1, chi=chi, hzero=False) for s in range(12)]

    def drift(tol):
        if batch and not tol:
            r = ffi.anneal_batch(probs, chi=chi)
        else:
            r = [ffi.anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi, jacobi_tol=tol) for p in probs]
        assert max(x.max_trunc for x in r) < 1e-24
        return np.sqrt(np.mean([(x.norm2 - 1.0) ** 2 for x in r]))

    assert drift(0.0) < 0.5 * drift(1e-13)
