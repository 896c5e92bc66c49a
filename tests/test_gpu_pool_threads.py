"""Calls from several threads at once share the pool of one-call memory: each gives what it gives alone."""
import threading

import numpy as np
import pytest

from tessera_b200 import ffi, instances, learned

pytestmark = pytest.mark.gpu


def test_threads_share_the_pool():
    p = instances.chain_range(n=17, dmax=2, seed=4, T=0.4, dt=0.1, chi=8, dist="normal", hzero=False)
    q = [instances.chain_range(n=n, dmax=1, seed=n, T=0.4, dt=0.1, chi=16) for n in (8, 9, 10)]
    a = np.random.default_rng(3).normal(size=(60, 50)) + 0j

    def session():
        s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=8)  # plain memory
        s.run(0, 2)
        e = s.sample(50, seed=2)[1].tolist()
        s.close()
        return e

    calls = [lambda: ffi.anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=8).expected_energy,
             lambda: [r.expected_energy for r in ffi.anneal_batch(q)],
             lambda: ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=1).expected_energy,
             lambda: learned.exact_ground(p)[0],
             lambda: ffi.sa_solve([p] + q, restarts=40, sweeps=20)[0].tolist(),
             lambda: ffi.svd(a)[1].tolist(), session]
    want = [f() for f in calls]
    wrong = []

    def work(k):
        for i in range(12):
            j = (i + k) % len(calls)
            got = calls[j]()
            if got != want[j]:
                wrong.append((k, j, got))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
