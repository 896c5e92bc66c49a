"""A resident complex128 theta is rotated by the same instructions alone and in a batch of its size class."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [40, 48, 56])
@pytest.mark.parametrize("from_end", [4, 5, 6])
def test_batch_and_single_give_the_same_bits(chi, from_end):
    """Theta of 2 chi rows and 2^(from_end + 1) columns (up to 2 chi): narrow ones leave a launch of their own
    fewer threads than a batch's, whose blocks are sized for 2 chi columns."""
    n = 16
    probs = [instances.chain_range(n=n, dmax=1, seed=s, T=2.0, dt=0.1, chi=chi) for s in range(2)]
    bond = n - from_end - 2
    p = probs[0]
    one = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi)
    two = ffi.Session.batch(probs, precision="c128")
    for s in (one, two):
        s.randomize(5, 6.0)
        s.run_gates(10, bond, bond + 1)
        assert s.sync().status == 0
    a = ffi.checkpoint_to_sites(one.save())[1]
    b = ffi.checkpoint_to_sites(two.save_instance(0))[1]
    one.close()
    two.close()
    assert 2 * a[bond].shape[0] == 2 * chi
    for i in (bond, bond + 1):
        assert a[i].shape == b[i].shape and np.array_equal(a[i], b[i]), i
