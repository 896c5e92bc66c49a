"""tessera_qa_exact_ground at the sizes where its table scan begins, on ties, self-loops and weights
that leave every pattern equal: the first minimum of the energies summed in edge order."""
import numpy as np
import pytest

from tessera_b200 import instances, learned

pytestmark = pytest.mark.gpu


def _first_minimum(p):
    x = np.arange(1 << p.n)
    s = [np.where((x >> i) & 1, 1.0, -1.0) for i in range(p.n)]
    e = np.zeros(1 << p.n)
    for i, j, w in zip(p.ei, p.ej, p.ew):
        e -= w * (s[i] * s[j])
    for i in range(p.n):
        e -= p.h[i] * s[i]
    k = int(np.argmin(e))  # first on ties
    return e[k], [1 if (k >> i) & 1 else -1 for i in range(p.n)]


@pytest.mark.parametrize("n", [15, 16, 17, 19])
@pytest.mark.parametrize("kind", ["random", "no_field", "integer", "loops", "flat", "last_bits"])
def test_first_minimum(n, kind):
    """Bit for bit: the energy is the same sum in the same order, the pattern its first minimum."""
    rng = np.random.Generator(np.random.PCG64(n))
    pairs = [(i, j) for i in range(n) for j in range(i + 1, n) if rng.random() < 0.5]
    if kind == "loops":
        pairs += [(3, 3), (n - 1, n - 1), (9, 2), (n - 1, 0)]
    w = rng.uniform(-1, 1, len(pairs))
    h = rng.uniform(-0.2, 0.2, n)
    if kind == "no_field":
        h = np.zeros(n)
    elif kind == "integer":  # many exact ties
        w, h = np.sign(w), np.zeros(n)
    elif kind == "flat":
        w, h = np.zeros(len(pairs)), np.zeros(n)
    elif kind == "last_bits":  # sums that differ in their last bits only
        w = np.where(np.arange(len(pairs)) % 2, 0.1, 0.3) * np.sign(w)
        h = 0.1 * np.sign(h)
    p = instances.Problem(h, np.array([a for a, _ in pairs]), np.array([b for _, b in pairs]), w)
    e, s = learned.exact_ground(p)
    e_ref, s_ref = _first_minimum(p)
    assert e == e_ref and list(s) == s_ref
