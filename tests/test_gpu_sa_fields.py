"""The annealing scorer's kept fields and FP32 screen, where they could differ from an FP64 test on a field
summed at the visit: long runs, couplings of many magnitudes that cancel, repeated pairs, scales outside FP32's
range.  Draw for draw against the oracle, as in test_gpu_sa.py."""
import numpy as np
import pytest

from oracle.oracle import Instance
from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _problem(n, p_edge, mag, seed, repeat=0):
    rng = np.random.Generator(np.random.PCG64(seed))
    edges = [(i, j) for i in range(n) for j in range(i + 1, n) if rng.random() < p_edge]
    edges += [edges[k] for k in rng.integers(0, len(edges), repeat)]
    w = rng.choice([-1.0, 1.0], len(edges)) * 10.0 ** rng.integers(-mag, mag + 1, len(edges))
    w[: len(w) // 2] *= rng.uniform(0.5, 1.0, len(w) // 2)
    ei, ej = (np.array([e[k] for e in edges], np.int64) for k in (0, 1))
    return instances.Problem(rng.uniform(-0.2, 0.2, n), ei, ej, w)


def _check(oracle, probs, restarts, sweeps, t0, t_end):
    en, spins = ffi.sa_solve(probs, restarts=restarts, sweeps=sweeps, t0=t0, t_end=t_end, seed=5)
    for b, p in enumerate(probs):
        inst = Instance(p.h, p.ei.astype(np.int32), p.ej.astype(np.int32), p.ew)
        s_o, e_o = oracle.sa_solve(inst, restarts, sweeps, t0=t0, t_end=t_end, seed=5, index=b)
        assert en[b] == e_o and list(spins[b]) == list(s_o), b


@pytest.mark.parametrize("mag", [0, 3, 8, 15])
def test_couplings_of_many_magnitudes(oracle, mag):
    """Temperatures between the smallest and the largest couplings, so that both kinds of energy change are
    undecided for a while; beyond 10^8 the large ones leave the small ones nothing but rounding."""
    probs = [_problem(n, 0.6, mag, 10 * mag + n) for n in (9, 24, 40)]
    probs.append(_problem(20, 0.5, mag, mag + 7, repeat=12))
    _check(oracle, probs, 20, 150, 10.0 ** mag, 10.0 ** -mag * 0.1)


def test_thousands_of_sweeps(oracle):
    _check(oracle, [_problem(16, 0.7, 2, 3), _problem(12, 0.6, 6, 4, repeat=5)], 6, 5000, 50.0, 1e-3)


@pytest.mark.parametrize("scale", [1e-300, 1e-42, 1e-36, 1e36, 1e39, 1e42, 1e300])
def test_scales_beyond_single_precision(oracle, scale):
    """A power of ten in couplings, fields and temperatures alike leaves the run what it was."""
    probs = [_problem(n, 0.6, 1, n) for n in (10, 30)]
    for p in probs:
        p.h, p.ew = p.h * scale, p.ew * scale
    _check(oracle, probs, 20, 60, 20.0 * scale, 0.05 * scale)
