"""The annealing scorer at the edges of its chain groups (8 lanes a chain, 16 chains a CTA) and of
its graph sizes, draw for draw against the oracle."""
import numpy as np
import pytest

from oracle.oracle import Instance
from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _problem(n, edges, rng):
    ei = np.array([e[0] for e in edges], np.int64)
    ej = np.array([e[1] for e in edges], np.int64)
    return instances.Problem(rng.uniform(-0.2, 0.2, n), ei, ej, rng.uniform(-1, 1, len(edges)))


@pytest.mark.parametrize("restarts,sweeps", [(1, 1), (15, 9), (17, 40), (300, 8)])
def test_sizes_match_the_oracle_draw_for_draw(oracle, restarts, sweeps):
    rng = np.random.Generator(np.random.PCG64(restarts))
    probs = [_problem(1, [], rng)]
    for n in (7, 8, 9, 64, 65):
        probs.append(_problem(n, [(i, j) for i in range(n) for j in range(i + 1, n) if rng.random() < 0.4], rng))
    probs.append(_problem(128, [(i, j) for i in range(128) for j in range(i + 1, 128)], rng))
    probs.append(_problem(6, [(0, 1), (1, 0), (0, 1), (2, 2), (3, 4), (4, 3)], rng))  # repeated pairs, a self-loop
    en, spins = ffi.sa_solve(probs, restarts=restarts, sweeps=sweeps, seed=3)
    for b, p in enumerate(probs):
        s_o, e_o = oracle.sa_solve(Instance(p.h, p.ei.astype(np.int32), p.ej.astype(np.int32), p.ew), restarts,
                                   sweeps, seed=3, index=b)
        assert en[b] == e_o and list(spins[b]) == list(s_o), (b, p.n)
