"""tessera_qa_svd's factors, formed on the device, at the edges of their 32 x 32 tiles, on rank-deficient
input and with either factor left out."""
import ctypes as C

import numpy as np
import pytest

from tessera_b200 import _lib, ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (1, 33), (33, 1), (31, 32), (32, 31), (65, 64), (37, 130), (130, 37),
                                   (257, 40)])
@pytest.mark.parametrize("rank", [None, 3])
def test_factors(shape, rank):
    """Isometries and a reconstruction to a few hundred roundings: 1e-12 x sqrt(size)."""
    rng = np.random.Generator(np.random.PCG64(shape[0] * 1000 + shape[1]))
    k = min(shape)
    a = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    if rank:
        r = min(rank, k)
        a = a[:, :r] @ (rng.normal(size=(r, shape[1])) + 1j * rng.normal(size=(r, shape[1])))
    u, s, vh = ffi.svd(a)
    ref = np.linalg.svd(a, compute_uv=False)
    tol = 1e-12 * np.sqrt(max(shape)) * np.linalg.norm(a)
    assert np.max(np.abs(s - ref)) < tol
    assert np.linalg.norm((u * s) @ vh - a) < tol
    live = np.linalg.norm(u, axis=0) > 0.5  # a sub-floor column with nothing left is zero
    g = u[:, live].conj().T @ u[:, live]
    assert np.linalg.norm(g - np.eye(live.sum())) < 1e-10
    assert live[ref > 1e-10 * ref[0]].all()
    big = ref > 1e-3 * ref[0]
    assert np.linalg.norm(vh[big] @ vh[big].conj().T - np.eye(big.sum())) < 1e-9


def test_either_factor_can_be_left_out():
    L = _lib.load()
    a = np.random.default_rng(1).normal(size=(40, 30)) + 0j
    u, s, vh = ffi.svd(a)
    for want_u, want_v in ((0, 0), (1, 0), (0, 1)):
        s2, u2, v2 = np.zeros(30), np.zeros((40, 30), complex), np.zeros((30, 30), complex)
        p = lambda x: x.view(np.float64).ctypes.data_as(_lib.c_double_p)  # noqa: E731
        assert L.tessera_qa_svd(p(a), 40, 30, p(s2), p(u2) if want_u else None, p(v2) if want_v else None) == 0
        assert np.array_equal(s2, s)
        assert np.array_equal(u2, u) if want_u else not u2.any()
        assert np.array_equal(v2, vh) if want_v else not v2.any()
