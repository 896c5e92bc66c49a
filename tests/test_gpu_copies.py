"""Host-to-device copies are ordered before the kernels that read them."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances, learned

pytestmark = pytest.mark.gpu


def test_set_params_reaches_the_bf16_weights():
    """The BF16 copy is made from the weights just set, every time: two weight vectors set in turn
    give the same two losses again and again.  The gradient's float atomics move the loss not at
    all and the loss is one block's sum, so the values repeat exactly; 1e-6 leaves room."""
    probs = [instances.dense_er(10, seed=s) for s in range(4)]
    net = learned.ScheduleGNN(hidden=64, layers=3, knots=16, seed=1)
    rng = np.random.Generator(np.random.PCG64(3))
    params = [(0.1 * rng.normal(size=net.param_count)).astype(np.float32) for _ in range(2)]
    tk = np.tile(np.linspace(0.0, 1.0, 16), (4, 1))
    ts = np.ones(40, np.float32)
    first = {}
    for _ in range(100):
        for k, p in enumerate(params):
            net.set_params(p)
            loss, _ = net.train_step(probs, tk, ts, lr=0.0)
            assert abs(loss - first.setdefault(k, loss)) < 1e-6 * abs(loss)
    assert abs(first[0] - first[1]) > 1e-4 * abs(first[0])
    net.close()


def test_load_reaches_the_kernels_that_run_next():
    """A checkpoint loaded and run at once gives the same state each time."""
    p = instances.chain_range(n=12, dmax=2, seed=3, T=0.4, dt=0.1, chi=64)
    s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=64)
    s.randomize(5)
    a = s.save()
    s.randomize(6)
    b = s.save()
    seen = {}
    for _ in range(10):
        for k, ck in enumerate((a, b)):
            s.load(ck)
            s.run_gates(2, 10, 12)
            assert s.save() == seen.setdefault(k, s.save())
    s.close()
