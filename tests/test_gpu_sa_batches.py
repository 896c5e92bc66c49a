"""The annealing scorer with the GPU full of chains: 4 lanes a chain, and on sparse graphs one thread a chain.
Draw for draw against the oracle, as in test_gpu_sa.py."""
import numpy as np
import pytest

from oracle.oracle import Instance
from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _problem(n, edges, rng):
    ei, ej = (np.array([e[k] for e in edges], np.int64) for k in (0, 1))
    return instances.Problem(rng.uniform(-0.2, 0.2, n), ei, ej, rng.uniform(-1, 1, len(edges)))


def _ring(n, rng, extra=()):
    return _problem(n, [(i, (i + 1) % n) for i in range(n)] + list(extra), rng)


def _dense(n, rng, extra=()):
    return _problem(n, [(i, j) for i in range(n) for j in range(i + 1, n)] + list(extra), rng)


@pytest.mark.parametrize("kind,count,restarts", [("sparse", 148, 256), ("sparse", 37, 1025), ("sparse", 147, 257),
                                                 ("dense", 148, 256), ("dense", 444, 32), ("dense", 458, 31)])
def test_full_batches_match_the_oracle_draw_for_draw(oracle, kind, count, restarts):
    rng = np.random.Generator(np.random.PCG64(count))
    make = _ring if kind == "sparse" else _dense
    repeats = [(0, 1), (1, 0), (2, 2), (3, 4), (4, 3)]
    probs = [make(n, rng) for n in (5, 9, 33, 64, 65, 128)] + [make(7, rng, repeats)]
    if kind == "dense":  # at the limit of shared memory: 199 KB of graph, too much beside 4 lanes' fields
        probs.append(_dense(128, rng, [(i, j) for i in range(60) for j in range(i + 1, 60)]))
    probs = (probs * (count // len(probs) + 1))[:count]
    en, spins = ffi.sa_solve(probs, restarts=restarts, sweeps=5, seed=9)
    for b in sorted({*range(8), count // 2, count - 1}):
        p = probs[b]
        inst = Instance(p.h, p.ei.astype(np.int32), p.ej.astype(np.int32), p.ew)
        s_o, e_o = oracle.sa_solve(inst, restarts, 5, seed=9, index=b)
        assert en[b] == e_o and list(spins[b]) == list(s_o), (b, p.n)
