"""Values that are not numbers: the column orders of every Jacobi kernel stay permutations of the columns
(a NaN norm once let the sort's padding in, whose indices lie beyond the matrix), so such input costs its
own result and nothing else."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 5), (70, 33), (113, 113), (200, 130), (300, 290), (520, 515)])
def test_svd_with_a_nan_column(shape):
    """The NaN column takes the last value, zero, and a zero column of u; the others are the SVD of the
    columns without it (1e-12 x sqrt(rows) as in test_gpu_svd_factors.py)."""
    rng = np.random.Generator(np.random.PCG64(shape[0]))
    a = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    bad = shape[1] // 2
    rest = np.delete(a, bad, axis=1)
    a[1, bad] = np.nan
    u, s, vh = ffi.svd(a)
    tol = 1e-12 * np.sqrt(shape[0]) * np.linalg.norm(rest)
    assert s[-1] == 0 and not u[:, -1].any()
    assert np.max(np.abs(s[:-1] - np.linalg.svd(rest, compute_uv=False))) < tol
    got = (u[:, :-1] * s[:-1]) @ np.delete(vh[:-1], bad, axis=1)
    assert np.linalg.norm(got - rest) < tol


@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("count,chi", [(1, 20), (2, 20), (1, 65), (2, 65), (2, 150)])
def test_overflowing_angles_keep_to_their_own_instance(precision, count, chi):
    """A gate angle beyond the largest double makes theta NaN: the update keeps one column, and a
    second session of the same shape that lives beside it is untouched by it, bit for bit."""
    n = 2 * int(np.ceil(np.log2(chi))) + 2

    def session(scale):
        probs = [instances.chain_range(n=n, dmax=1, seed=s, T=2.0, dt=0.1, chi=chi) for s in range(count)]
        for p in probs:
            p.ew, p.sb = p.ew * scale, p.sb * scale
        if count > 1:
            s = ffi.Session.batch(probs, precision=precision)
        else:
            p = probs[0]
            s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi, precision=precision)
        s.randomize(3, chi / 4.0)
        return s

    bond = n // 2 - 1
    good, bad = session(1.0), session(1e200)
    before = [good.save_instance(b) for b in range(count)]
    bad.run_gates(10, bond, bond + 1)
    bad.sync()
    for b in range(count):
        assert ffi.checkpoint_to_sites(bad.save_instance(b))[1][bond].shape[2] == 1
    bad.close()
    assert [good.save_instance(b) for b in range(count)] == before
    good.close()
