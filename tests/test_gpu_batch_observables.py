"""A batch's observables, taken together, are the single runs' to the last bit: the same tiles summed
in the same order, one CTA per instance instead of a grid per instance."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("shapes", [[(1, 1), (2, 2), (5, 4), (9, 16), (10, 32), (11, 31)], [(12, 40)] * 33])
def test_batch_observables_equal_single_runs(precision, shapes):
    probs = [instances.chain_range(n=n, dmax=min(2, max(1, n - 1)), seed=k, T=0.3, dt=0.1, chi=chi, hzero=False)
             for k, (n, chi) in enumerate(shapes)]
    got = ffi.anneal_batch(probs, precision=precision)
    for k in sorted({0, 1, len(probs) // 2, len(probs) - 1}):
        p, g = probs[k], got[k]
        r = ffi.anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=p.chi, precision=precision)
        assert list(g.spins) == list(r.spins)
        assert (g.energy, g.expected_energy, g.prob, g.norm2) == (r.energy, r.expected_energy, r.prob, r.norm2)
        assert np.array_equal(g.z_expect, r.z_expect) and np.array_equal(g.entropy, r.entropy)
