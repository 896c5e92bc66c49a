"""The standalone SVD's left factor is an isometry to the tolerance its Jacobi stops at."""
import numpy as np
import pytest

from tessera_b200 import ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(20, 20), (64, 64), (112, 100), (200, 200), (320, 320), (100, 300), (600, 560)])
@pytest.mark.parametrize("graded", [False, True])
def test_inner_products_stop_at_the_tolerance(shape, graded):
    """|u_p^H u_q| is at most tol = max(2e-14, 4 sqrt(rows) 2^-52) when the last sweep ends, plus the rounding
    of the test's own products, sqrt(rows) 2^-53 at most here: 1.5 tol."""
    rng = np.random.Generator(np.random.PCG64(shape[0]))
    a = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    if graded:
        a = a * np.exp(-np.arange(shape[1]) / (shape[1] / 6.0))
    u, s, vh = ffi.svd(a)
    g = u.conj().T @ u
    tol = max(2e-14, 4.0 * np.sqrt(shape[0]) * 2.0 ** -52)
    assert np.max(np.abs(g - np.eye(min(shape)))) < 1.5 * tol
    assert np.linalg.norm((u * s) @ vh - a) < 1e-12 * np.linalg.norm(a)
