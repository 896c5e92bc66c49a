"""The state-vector anneal at the edges of its pass plan: one tile (n = 12), groups of one to seven
targets above it (13..19), two groups (20, 21), against the same evolution in torch on the device."""
import numpy as np
import pytest
import torch

from tessera_b200 import ffi, instances

pytestmark = pytest.mark.gpu


def _evolve(p, mode):
    n, dev = p.n, "cuda"
    x = torch.arange(1 << n, device=dev)
    z = [(1 - 2 * ((x >> i) & 1)).double() for i in range(n)]
    zz = torch.zeros(1 << n, dtype=torch.float64, device=dev)
    for i, j, w in zip(p.ei.tolist(), p.ej.tolist(), p.ew.tolist()):
        zz -= w * z[i] * z[j]
    full = zz - sum(float(p.h[i]) * z[i] for i in range(n))
    psi = torch.full((1 << n,), 2.0 ** (-0.5 * n), dtype=torch.complex128, device=dev)

    def gates(psi, f):
        for i in range(n):
            g = f(i)
            v = psi.reshape(-1, 2, 1 << i)
            psi = torch.stack([g[0][0] * v[:, 0] + g[0][1] * v[:, 1], g[1][0] * v[:, 0] + g[1][1] * v[:, 1]], 1).reshape(-1)
        return psi

    ent = []
    for a, b in zip(p.sa.tolist(), p.sb.tolist()):
        if mode == 0:
            ph = torch.exp(-0.5j * p.dt * b * full)
            c, s = np.cos(a * p.dt), np.sin(a * p.dt)
            psi = gates(psi * ph, lambda i: [[c, 1j * s], [1j * s, c]]) * ph
        else:
            def half(i):
                nx, nz = -a, -b * p.h[i]
                r = np.hypot(nx, nz)
                c, s = np.cos(0.5 * p.dt * r), (np.sin(0.5 * p.dt * r) / r if r else 0.0)
                return [[c - 1j * s * nz, -1j * s * nx], [-1j * s * nx, c + 1j * s * nz]]
            psi = gates(gates(psi, half) * torch.exp(-1j * p.dt * b * zz), half)
        m = psi.reshape(-1, 2)
        lam = np.clip(np.linalg.eigvalsh((m.T @ m.conj()).cpu().numpy()), 0, 1)
        ent.append(-sum(v * np.log2(v) for v in lam if v > 1e-12))
    return psi.cpu().numpy(), np.array(ent)


@pytest.mark.parametrize("n", [11, 12, 13, 14, 15, 16, 17, 19, 20, 21])
@pytest.mark.parametrize("mode", [0, 1])
def test_pass_plans(n, mode):
    """Six steps of gates and phases: 6 n roundings of 1e-16 per amplitude, 1e-13 of the state's norm;
    the entropy, of order 0.1, to 1e-11."""
    p = instances.chain_range(n=n, dmax=2, seed=n, T=0.6, dt=0.1, chi=1, dist="normal", hzero=False)
    g = ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=mode, want_state=True)
    psi, ent = _evolve(p, mode)
    assert np.linalg.norm(g.state - psi) < 1e-13
    assert np.max(np.abs(g.entropy - ent)) < 1e-11
    assert abs(g.norm2 - 1) < 1e-12


def test_many_steps_share_gate_and_entropy_launches():
    """More sweeps than one gate launch makes (256): every step's entropy is there."""
    p = instances.chain_range(n=6, dmax=1, seed=2, T=60.0, dt=0.1, chi=1, dist="normal", hzero=False)
    g = ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=1, want_state=True)
    psi, ent = _evolve(p, 1)
    assert np.linalg.norm(g.state - psi) < 1e-11
    assert np.max(np.abs(g.entropy - ent)) < 1e-10
