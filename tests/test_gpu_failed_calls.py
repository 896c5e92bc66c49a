"""Calls whose device memory comes from the library's pool, with the allocation made to fail: an error, all
memory and streams back, and the next call right."""
import numpy as np
import pytest

from tessera_b200 import _lib, ffi, instances, learned

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    L = _lib.load()
    yield L
    L.tessera_qa_debug_fail_allocations(0, 0)


def _calls():
    p = instances.chain_range(n=16, dmax=2, seed=4, T=0.4, dt=0.1, chi=8, dist="normal", hzero=False)
    a = np.random.default_rng(3).normal(size=(40, 30)) + 0j
    s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=8)
    s.run(0, 2)
    s.sample(4, seed=1)  # the environments stay with the session
    return {
        "sv_0": lambda: ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=0).expected_energy,
        "sv_1": lambda: ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=1).expected_energy,
        "ground": lambda: learned.exact_ground(p)[0],
        "sa": lambda: float(ffi.sa_solve([p], restarts=4, sweeps=10)[0][0]),
        "sample": lambda: s.sample(5, seed=2)[1].tolist(),
        "svd_workspace": lambda: ffi.svd(a)[1].tolist(),
    }, s


def test_a_failed_allocation_ends_the_call_alone(lib):
    import torch
    calls, s = _calls()
    want = {k: f() for k, f in calls.items()}
    for name, f in calls.items():
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        for _ in range(3):
            lib.tessera_qa_debug_fail_allocations(1 if name == "svd_workspace" else 0, 1)
            with pytest.raises(_lib.EngineError) as err:
                f()
            assert "out of memory" in str(err.value), name
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free0, name
        assert f() == want[name], name
    s.close()


def test_a_network_that_could_not_grow_still_takes_a_smaller_batch(lib):
    small, large = ([instances.dense_er(n, n, T=1.0, dt=0.1, chi=8) for n in ns] for ns in ((5, 6), (7, 8, 9, 10)))
    net = learned.ScheduleGNN(hidden=16, layers=2, knots=8, seed=2)
    want = net.forward(small)
    lib.tessera_qa_debug_fail_allocations(0, 1)
    with pytest.raises(_lib.EngineError) as err:
        net.forward(large)
    assert "out of memory" in str(err.value)
    got = net.forward(small)
    for a, b in zip(got, want):  # the messages of a node are summed in no fixed order: a few FP32 roundings
        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)
    net.close()
