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


@pytest.mark.parametrize("n,chi,dmax", [(2, 2, 1), (3, 3, 2), (5, 4, 2), (8, 5, 1), (9, 16, 2), (10, 17, 1),
                                        (10, 32, 2), (11, 32, 1), (12, 47, 1), (12, 56, 1)])
def test_rank_revealing_lq_leaves_the_anneal_alone(n, chi, dmax):
    """Small theta with and without the LQ in front of the resident Jacobi, from a product state (rank 1)
    through growing ranks, wide and tall theta at the ends of the chain.  <H>, <Z> and the entropy agree to
    1e-9, a thousand updates' worth of rounding at 1e-12, plus what truncation amplifies: ten times the
    change that 4 ulps on the inputs make to the run without the LQ."""
    p = instances.chain_range(n=n, dmax=dmax, seed=n, T=0.8, dt=0.1, chi=chi, hzero=False)

    def run(precondition, eps=0.0):
        r = ffi.anneal(p.h * (1 + eps), p.ei, p.ej, p.ew * (1 + eps), p.sa, p.sb * (1 + eps), dt=p.dt, chi=chi,
                       jacobi_precondition=precondition)
        assert r.status == 0
        return [np.atleast_1d(x) for x in (r.expected_energy, r.z_expect, r.entropy, r.norm2, r.max_trunc)]

    ref = run(2)
    moved = [run(2, eps) for eps in (4e-16, -4e-16, 8e-16)]
    for k, (x, y) in enumerate(zip(run(0), ref)):
        own = max(np.max(np.abs(m[k] - y)) for m in moved)
        assert np.max(np.abs(x - y)) < 1e-9 + 10 * own, k
