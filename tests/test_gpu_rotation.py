"""The complex128 rotation by itself: one sweep over a theta whose columns meet in pairs only."""
import struct

import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _checkpoint(sites):
    n = len(sites)
    dims = [s.shape[0] for s in sites] + [sites[-1].shape[2]]
    head = b"TQMPSv1\0" + struct.pack("<IIQQ", n, 0, 0, 0) + np.array(dims, np.int32).tobytes()
    head += b"\0" * (-len(head) % 8)
    return head + b"".join(np.ascontiguousarray(s, np.complex128).tobytes() for s in sites)


@pytest.mark.parametrize("scale", [1.0, 1e60])
@pytest.mark.parametrize("chi", [2, 8, 32, 56, 64, 128])
def test_one_rotation_annihilates_to_rounding(chi, scale):
    """theta = A C with A an embedding and C of 2 x 2 blocks, a weightless gate, one sweep of the Jacobi
    without the LQ: each pair of columns is rotated once.  With F^2 = |w_p|^2 + |w_q|^2 and r = 2^-53, what may
    be left of w_p^H w_q is 4 r F^2 from the sums, 8 r |gamma| <= 4 r F^2 from s and c, and 2 x 8 r F^2 from
    the rounding of both rotated columns: 24 r F^2, here 64 r F^2.  (An angle good to 1e-7 leaves 1e-7.)
    """
    rng = np.random.Generator(np.random.PCG64(chi))
    half = chi.bit_length()  # sites on each side that carry the bond up to chi
    n = 2 * half
    p = instances.chain_nn(n=n, seed=1, T=1.0, dt=0.1, chi=chi)
    p.ew[:] = 0.0
    sites = []
    for i in range(n):
        left = min(chi, 2 ** min(i, n - i))
        right = min(chi, 2 ** min(i + 1, n - i - 1))
        sites.append(np.zeros((left, 2, right), complex))
        sites[-1][np.arange(min(left, right)), 0, np.arange(min(left, right))] = 1.0
    bond = half - 1
    m = sites[bond].shape[2]
    blocks = rng.normal(size=(m // 2, 2, 2)) + 1j * rng.normal(size=(m // 2, 2, 2))
    a = np.zeros((2 * sites[bond].shape[0], m), complex)
    a[rng.permutation(a.shape[0])[:m], np.arange(m)] = 1.0
    c = np.zeros((m, 2 * sites[bond + 1].shape[2]), complex)
    cols = rng.permutation(c.shape[1])[:m]
    for k in range(m // 2):
        c[2 * k:2 * k + 2, cols[2 * k:2 * k + 2]] = blocks[k] * scale
    sites[bond] = a.reshape(sites[bond].shape)
    sites[bond + 1] = c.reshape(m, 2, -1)
    s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi, jacobi_max_sweeps=1, jacobi_precondition=2)
    s.load(_checkpoint(sites))
    s.run_gates(1, bond, bond + 1)
    s.sync()
    u = ffi.checkpoint_to_sites(s.save())[1][bond]
    s.close()
    u = u.reshape(-1, u.shape[2])
    theta = a @ c
    assert u.shape == (theta.shape[0], m)
    sv = np.linalg.norm(u.conj().T @ theta, axis=1)
    w = (u * sv) / scale
    g = np.abs(w.conj().T @ w)
    nrm = np.sum(np.abs(w) ** 2, axis=0)
    off = g - np.diag(np.diag(g))
    assert np.max(off / (nrm[:, None] + nrm[None, :])) < 64 * 2.0 ** -53
    assert np.max(np.abs(np.sqrt(nrm) - np.linalg.svd(theta / scale, compute_uv=False)[:m][np.argsort(np.argsort(-nrm))])) \
        < 64 * 2.0 ** -53 * np.max(np.sqrt(nrm))
