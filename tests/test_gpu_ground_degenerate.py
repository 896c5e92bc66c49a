"""The exact ground state where the second pass of the table scan sums most patterns, at the splits of its
chunks over CTAs (8 parts up to n = 23, 4 beyond): the first minimum in pattern order."""
import numpy as np
import pytest

from tessera_b200 import instances, learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 17, 22, 23, 24, 25])
@pytest.mark.parametrize("kind", ["zero", "last_pair", "first_pair", "last_field"])
def test_first_minimum_of_a_degenerate_instance(n, kind):
    """Bit i of a pattern set means s_i = +1, so the first minimum has every free spin down."""
    ei, ej = np.triu_indices(n, 1)
    p = instances.Problem(np.zeros(n), ei.astype(np.int64), ej.astype(np.int64), np.zeros(len(ei)))
    want, energy = -np.ones(n, np.int8), 0.0
    if kind == "last_pair":  # antiparallel: the lower of the two spins up
        p.ew[-1], energy = -1.5, -1.5
        want[n - 2] = 1
    elif kind == "first_pair":
        p.ew[0], energy = -0.5, -0.5
        want[0] = 1
    elif kind == "last_field":
        p.h[-1], energy = 2.0, -2.0
        want[n - 1] = 1
    e, spins = learned.exact_ground(p)
    assert e == energy and list(spins) == list(want)
