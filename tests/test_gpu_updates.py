"""One two-site update of a saturated random MPS against numpy's SVD, at the edges of the Jacobi
kernels' size classes and block widths."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _truncated_theta(sites, bond, theta_angle, chi):
    """exp(-i angle Z Z) on sites bond, bond + 1, truncated to chi by numpy's SVD."""
    a, c = sites[bond], sites[bond + 1]
    t = np.einsum("asc,ctb->astb", a, c)
    ph = np.exp(-1j * theta_angle * np.array([[1.0, -1.0], [-1.0, 1.0]]))
    th = (t * ph[None, :, :, None]).reshape(2 * a.shape[0], 2 * c.shape[2])
    u, s, vh = np.linalg.svd(th, full_matrices=False)
    return (u[:, :chi] * s[:chi]) @ vh[:chi]


@pytest.mark.parametrize("count,chi,block", [(2, 57, 0), (3, 64, 4), (2, 65, 0), (2, 127, 8), (2, 129, 0),
                                             (2, 201, 4), (2, 255, 0), (1, 57, 0), (1, 65, 0), (1, 129, 0),
                                             (1, 255, 0), (1, 129, 4), (1, 31, 0), (2, 47, 0)])
def test_update_matches_numpy(count, chi, block):
    """Graded spectra (decay chi / 5): neighbouring singular values at the cut differ by about
    s / (chi / 10), so two accurate SVDs agree on the truncated theta to a few hundred rounding
    errors of ||theta||: 512 x 2^-52 x 100 = 1e-11."""
    n = 14 if chi <= 64 else 16 if chi <= 128 else 18
    probs = [instances.chain_range(n=n, dmax=1, seed=s, T=2.0, dt=0.1, chi=chi) for s in range(count)]
    if count > 1:
        s = ffi.Session.batch(probs, precision="c128", jacobi_block=block)
    else:
        p = probs[0]
        s = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=chi, jacobi_block=block)
    s.randomize(5, chi / 5.0)
    before = [ffi.checkpoint_to_sites(s.save_instance(b))[1] for b in range(count)]
    bond = n // 2 - 1
    s.run_gates(10, bond, bond + 1)
    r = s.sync()
    assert r.status == 0
    for b, p in enumerate(probs):
        after = ffi.checkpoint_to_sites(s.save_instance(b))[1]
        a, c = after[bond], after[bond + 1]
        got = np.einsum("asc,ctb->astb", a, c).reshape(2 * a.shape[0], 2 * c.shape[2])
        ref = _truncated_theta(before[b], bond, -p.sb[10] * p.ew[bond] * p.dt, chi)
        assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref), (chi, b)
        iso = a.reshape(-1, a.shape[2])
        assert np.linalg.norm(iso.conj().T @ iso - np.eye(a.shape[2])) < 1e-11
    s.close()
