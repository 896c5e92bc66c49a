"""jacobi_block = 16 in complex128 batches: column-pair blocks of that width up to 256 rows (32 columns in
registers, 16 streamed), of 8 beyond."""
import numpy as np
import pytest

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [57, 63, 64, 65, 100, 127, 128, 129])
@pytest.mark.parametrize("precondition", [0, 2])
def test_update_matches_numpy(chi, precondition):
    """As test_gpu_updates.py: graded spectra, 512 x 2^-52 x 100 = 1e-11 of the truncated theta's norm."""
    n = 14 if chi <= 64 else 16
    probs = [instances.chain_range(n=n, dmax=1, seed=s, T=2.0, dt=0.1, chi=chi) for s in range(2)]
    s = ffi.Session.batch(probs, precision="c128", jacobi_block=16, jacobi_precondition=precondition)
    s.randomize(5, chi / 5.0)
    before = [ffi.checkpoint_to_sites(s.save_instance(b))[1] for b in range(2)]
    bond = n // 2 - 1
    s.run_gates(10, bond, bond + 1)
    assert s.sync().status == 0
    for b, p in enumerate(probs):
        a, c = before[b][bond], before[b][bond + 1]
        t = np.einsum("asc,ctb->astb", a, c)
        ang = -p.sb[10] * p.ew[bond] * p.dt
        t = t * np.exp(-1j * ang * np.array([[1.0, -1.0], [-1.0, 1.0]]))[None, :, :, None]
        u, sv, vh = np.linalg.svd(t.reshape(2 * a.shape[0], 2 * c.shape[2]), full_matrices=False)
        ref = (u[:, :chi] * sv[:chi]) @ vh[:chi]
        a, c = ffi.checkpoint_to_sites(s.save_instance(b))[1][bond:bond + 2]
        got = np.einsum("asc,ctb->astb", a, c).reshape(2 * a.shape[0], 2 * c.shape[2])
        assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref)
        iso = a.reshape(-1, a.shape[2])
        assert np.linalg.norm(iso.conj().T @ iso - np.eye(a.shape[2])) < 1e-11
    s.close()
