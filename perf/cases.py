"""Measured cases: the calls a user of this framework makes, with the sizes they make them at.

Every case is one pass through a public entry point (`tessera_b200.ffi`, `tessera_b200.learned`):

* ``anneal`` -- one instance through `ffi.anneal` (or the drop-in `ffi.quantum_anneal`);
* ``batch``  -- many small instances through `ffi.anneal_batch`, as labelling and solving do;
* ``gates``  -- a window of two-site updates on saturated bonds of a device-resident session,
  through the host-buffer call `Session.run_host`, then a checkpoint;
* ``sv``     -- the exact state-vector anneal, `ffi.sv_anneal`;
* ``svd``    -- `ffi.svd`;
* ``gnn``    -- one training step of the schedule network;
* ``sa``, ``ground`` -- the scorers `ffi.sa_solve` and `learned.exact_ground`.

``exact`` restates each of them in plain numpy or torch in 64 bits.  An MPS is only defined up to
a phase per Schmidt vector, so sessions return the state itself (all 2^n amplitudes contracted
from the checkpoint) and `ffi.svd`'s factors come with the first row of u made real.
"""
import math

import numpy as np
import torch

from tessera_b200 import ffi, instances, learned


# ------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------
def listed():
    return [
        # the drop-in symbol on the reference tests' scale: one tiny exact anneal, all latency
        dict(name="legacy_n6", kind="anneal", legacy=True, graph="chain", n=6, dmax=2, chi=8, steps=30,
             stop=30, dt=0.1, precision="c128"),
        # the n=16 chain study: nearest-neighbour chain at chi=32, the first steps of its 400 in one
        # complex128 call
        dict(name="chain16_chi32", kind="anneal", legacy=False, graph="chain", n=16, dmax=1, chi=32, steps=400,
             stop=40, dt=0.05, precision="c128"),
        # labelling: small dense instances at chi=32, one batch of schedule candidates, complex128
        dict(name="batch_er10_c128", kind="batch", count=160, n_lo=8, n_hi=10, chi=32, steps=6, dt=0.1,
             precision="c128"),
        # the solve batch: held-out dense instances of a dozen spins at chi=32 in complex64
        dict(name="batch_er13_c64", kind="batch", count=296, n_lo=12, n_hi=13, chi=32, steps=2, dt=0.1,
             precision="c64"),
        # the headline: saturated chi=256 updates of a full batch, one instance per SM
        dict(name="gates_chi256_c128", kind="gates", count=148, n=20, dmax=4, chi=256, slots=1, decay=48.0,
             precision="c128"),
        # the ragged study's larger cap: chi=128 updates of a batch in complex64
        dict(name="gates_chi128_c64", kind="gates", count=148, n=18, dmax=4, chi=128, slots=4, decay=32.0,
             precision="c64"),
        # the plain engine: one instance at chi=256, then its observables
        dict(name="single_chi256_c128", kind="gates", count=1, n=20, dmax=4, chi=256, slots=8, decay=48.0,
             precision="c128"),
        # the exact state vector that runs are checked against, engine splitting
        dict(name="sv_n22", kind="sv", n=22, dmax=2, steps=40, dt=0.05, mode=1),
        # the standalone SVD on host buffers
        dict(name="svd_320", kind="svd", rows=320, cols=320),
        # one mini-batch of schedule-network training at its default size
        dict(name="gnn_train_32", kind="gnn", count=32, n_lo=8, n_hi=12, hidden=64, layers=3, knots=16),
        # best-known energies beyond brute force
        dict(name="sa_n48", kind="sa", count=8, n=48, restarts=512, sweeps=500),
        # exact ground energies, which labels and solves are scored against
        dict(name="ground_n22", kind="ground", n=22),
    ]


def _log(rng, lo, hi):
    """A whole number in lo..hi, uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["anneal", "anneal", "batch", "batch", "gates", "gates", "gates", "sv", "svd", "gnn", "sa",
                       "ground"])
    if kind == "anneal":
        legacy = rng.random() < 0.3
        n = rng.randint(5, 10 if legacy else 16)
        if n <= 8 and rng.random() < 0.5:
            steps = rng.randint(6, 12)
            return dict(kind=kind, legacy=legacy, graph="er", n=n, dmax=0, chi=16, steps=steps, stop=steps, dt=0.1,
                        precision="c128")
        if n <= 10:  # a whole short anneal; bonds never truncate
            dmax = rng.choice([1, 1, 2])
            steps = rng.randint(20, 60) // dmax
            return dict(kind=kind, legacy=legacy, graph="chain", n=n, dmax=dmax, chi=32, steps=steps, stop=steps,
                        dt=0.1 if legacy else 0.05, precision="c128")
        if n <= 12:  # the precision study's exact chi=64 chains
            dmax = rng.randint(1, 3)
            steps = rng.randint(20, 40) // dmax
            return dict(kind=kind, legacy=False, graph="chain", n=n, dmax=dmax, chi=64, steps=steps, stop=steps,
                        dt=0.05, precision="c128")
        return dict(kind=kind, legacy=False, graph="chain", n=n, dmax=1, chi=32, steps=400, stop=rng.randint(15, 40),
                    dt=0.05, precision="c128")
    if kind == "batch":
        if rng.random() < 0.5:
            lo = rng.randint(6, 9)
            return dict(kind=kind, count=_log(rng, 16, 296), n_lo=lo, n_hi=rng.randint(lo, 10), chi=32,
                        steps=rng.randint(3, 6), dt=0.1, precision="c128")
        lo = rng.randint(10, 13)
        return dict(kind=kind, count=_log(rng, 16, 296), n_lo=lo, n_hi=rng.randint(lo, 13), chi=32,
                    steps=2, dt=0.1, precision="c64")
    if kind == "gates":
        which = rng.random()
        if which < 0.34:
            chi = _log(rng, 136, 256)
            return dict(kind=kind, count=_log(rng, 16, 148), n=20, dmax=rng.randint(2, 4), chi=chi, slots=1,
                        decay=float(max(24, chi // 5)), precision="c128")
        if which < 0.67:
            chi = _log(rng, 72, 256)
            return dict(kind=kind, count=_log(rng, 16, 148), n=20 if chi > 128 else 18, dmax=rng.randint(2, 4),
                        chi=chi, slots=rng.randint(1, 2), decay=float(max(24, chi // 4)), precision="c64")
        chi = _log(rng, 64, 256)
        return dict(kind=kind, count=1, n=20 if chi > 128 else 18, dmax=rng.randint(2, 4), chi=chi,
                    slots=rng.randint(4, 8), decay=float(max(24, chi // 5)), precision="c128")
    if kind == "sv":
        return dict(kind=kind, n=rng.randint(8, 22), dmax=rng.randint(1, 3), steps=rng.randint(20, 40), dt=0.05,
                    mode=rng.randint(0, 1))
    if kind == "svd":
        return dict(kind=kind, rows=_log(rng, 24, 320), cols=_log(rng, 24, 320))
    if kind == "gnn":
        lo = rng.randint(6, 16)
        return dict(kind=kind, count=_log(rng, 4, 64), n_lo=lo, n_hi=lo + rng.randint(0, 6),
                    hidden=rng.choice([32, 64]), layers=rng.randint(2, 3), knots=16)
    if kind == "sa":
        return dict(kind=kind, count=_log(rng, 1, 16), n=rng.randint(20, 64), restarts=_log(rng, 40, 512),
                    sweeps=_log(rng, 200, 500))
    return dict(kind=kind, n=rng.randint(10, 23))


# ------------------------------------------------------------------------------------
# inputs (made from the seed alone)
# ------------------------------------------------------------------------------------
def _schedule(steps):
    s = np.arange(steps, dtype=np.float64) / (steps - 1)
    return 1.0 - s, s


def _problem(graph, n, dmax, steps, dt, chi, rng):
    """Chain with couplings to distance dmax (J ~ N(0, 1), h ~ N(0, 1/2)) or a dense Erdos-Renyi
    graph (p = 1/2, J ~ U(-1, 1), h ~ U(-0.2, 0.2)), under the linear schedule."""
    if graph == "chain":
        pairs = [(i, i + d) for i in range(n) for d in range(1, dmax + 1) if i + d < n]
        ew = rng.normal(0.0, 1.0, len(pairs))
        h = rng.normal(0.0, 0.5, n)
    else:
        pairs = [(i, j) for i in range(n) for j in range(i + 1, n) if rng.random() < 0.5] or [(0, 1)]
        ew = rng.uniform(-1.0, 1.0, len(pairs))
        h = rng.uniform(-0.2, 0.2, n)
    sa, sb = _schedule(max(steps, 2))
    ei, ej = np.array([p[0] for p in pairs], np.int64), np.array([p[1] for p in pairs], np.int64)
    return instances.Problem(h, ei, ej, ew, sa, sb, dt, chi)


def _problems(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 17]))
    k = case["kind"]
    if k == "anneal":
        return [_problem(case["graph"], case["n"], case["dmax"], case["steps"], case["dt"], case["chi"], rng)]
    if k in ("batch", "gnn"):
        return [_problem("er", case["n_lo"] + b % (case["n_hi"] - case["n_lo"] + 1), 0, case.get("steps", 2),
                         case.get("dt", 0.1), case.get("chi", 32), rng) for b in range(case["count"])]
    if k == "gates":
        return [_problem("chain", case["n"], case["dmax"], 41, 0.1, case["chi"], rng) for _ in range(case["count"])]
    if k == "sv":
        return [_problem("chain", case["n"], case["dmax"], case["steps"], case["dt"], 1, rng)]
    if k == "sa":
        return [_problem("er", case["n"], 0, 2, 0.1, 1, rng) for _ in range(case["count"])]
    return [_problem("er", case["n"], 0, 2, 0.1, 1, rng)]


def _window(case):
    """The two-site slots of a session case: from the first gate of the middle edge on, where every
    bond that the window touches is at its cap."""
    n, dmax = case["n"], case["dmax"]
    first = sum(2 * d - 1 for i in range(n // 2 - 2) for d in range(1, dmax + 1) if i + d < n)
    return first, first + case["slots"]


def _matrix(case, seed):
    """A matrix with a graded spectrum exp(-8 k / K), as a bond's Schmidt values fall."""
    rng = np.random.Generator(np.random.PCG64([seed, 23]))
    r, c = case["rows"], case["cols"]
    k = min(r, c)
    u = np.linalg.qr(rng.normal(size=(r, k)) + 1j * rng.normal(size=(r, k)))[0]
    v = np.linalg.qr(rng.normal(size=(c, k)) + 1j * rng.normal(size=(c, k)))[0]
    return (u * np.exp(-8.0 * np.arange(k) / k)) @ v.conj().T


def _gnn_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 29]))
    probs = _problems(case, seed)
    knots = np.sort(rng.random((case["count"], case["knots"])), axis=1)
    knots[:, 0], knots[:, -1] = 0.0, 1.0
    spins = (rng.random(sum(p.n for p in probs)) < 0.5).astype(np.float32)
    return probs, knots.astype(np.float32), spins, _gnn_params(case, rng)


def prepare(case, seed):
    k = case["kind"]
    if k == "svd":
        return dict(case=case, a=_matrix(case, seed))
    if k == "gnn":
        probs, knots, spins, params = _gnn_inputs(case, seed)
        net = learned.ScheduleGNN(hidden=case["hidden"], layers=case["layers"], knots=case["knots"], seed=1)
        net.set_params(params)
        torch.cuda.synchronize()  # the weights are in place before their BF16 copy is made again
        net.set_params(params)
        return dict(case=case, probs=probs, net=net, knots=knots, spins=spins)
    probs = _problems(case, seed)
    state = dict(case=case, probs=probs, seed=seed)
    if k == "gates":
        if case["count"] == 1:
            p = probs[0]
            state["session"] = ffi.Session(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=p.chi,
                                           precision=case["precision"])
        else:
            state["session"] = ffi.Session.batch(probs, precision=case["precision"])
    return state


# ------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------
def _dense(sites):
    """The 2^n amplitudes of an MPS on the GPU; bit i of the index is the physical index of site i."""
    v = torch.ones(1, 1, dtype=torch.complex128, device="cuda")
    for t in sites:
        t = torch.tensor(t, device="cuda")
        w = (v @ t.reshape(t.shape[0], -1)).reshape(v.shape[0], 2, t.shape[2])
        v = w.permute(1, 0, 2).reshape(-1, t.shape[2])
    return v[:, 0].contiguous()


def _results(rs, precision):
    """What an anneal returns, over the instances of a call (numbers: per instance the energies, the
    readout's probability, the norm, the discarded weight and <Z> of every spin); complex64 runs
    carry 32-bit accuracy."""
    f = np.float32 if precision == "c64" else np.float64
    return {"spins": np.concatenate([r.spins for r in rs]),
            "numbers": np.concatenate([np.append([r.energy, r.expected_energy, r.prob, r.norm2, r.max_trunc],
                                                 r.z_expect) for r in rs]).astype(f),
            "entropy": np.concatenate([r.entropy for r in rs]).astype(f)}


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "svd":
        u, s, vh = ffi.svd(state["a"])
        ph = u[0] / np.abs(u[0])
        return {"u": u * ph.conj(), "s": s, "vh": vh * ph[:, None]}
    if k == "gnn":
        loss, g = state["net"].train_step(state["probs"], state["knots"], state["spins"], lr=1e-4, want_grads=True)
        return {"loss": np.array([loss], np.float32), "grads": g}
    probs = state["probs"]
    p = probs[0]
    if k == "anneal":
        if case["legacy"]:
            m = ffi.Ising(list(p.h), list(zip(p.ei, p.ej, p.ew)))
            r = ffi.quantum_anneal(m, ffi.Schedule(list(p.sa), list(p.sb)), case["chi"])
            return {"spins": r.spins, "energy": r.energy, "entropy": r.entropy}
        return _results([ffi.anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, chi=p.chi,
                                    precision=case["precision"], step_end=case["stop"])], case["precision"])
    if k == "batch":
        return _results(ffi.anneal_batch(probs, precision=case["precision"]), case["precision"])
    if k == "gates":
        s = state["session"]
        s.randomize(state["seed"], case["decay"])
        r = s.run_host(probs, 20, *_window(case))
        wide = case["precision"] == "c128"
        out = {"kept": np.array([1.0 - r.max_trunc], np.float64 if wide else np.float32)}
        if case["count"] == 1:
            spins = np.zeros(case["n"], np.int8)
            o = s.observe(spins)
            out |= {"spins": spins, "numbers": np.array([o.energy, o.expected_energy, o.prob, o.norm2])}
        for b in sorted({0, case["count"] - 1}):
            psi = _dense(ffi.checkpoint_to_sites(s.save_instance(b))[1])
            out["state%d" % (b > 0)] = psi if wide else psi.to(torch.complex64)
        return out
    if k == "sv":
        r = ffi.sv_anneal(p.h, p.ei, p.ej, p.ew, p.sa, p.sb, dt=p.dt, mode=case["mode"])
        return {"spins": r.spins, "sign_spins": r.sign_spins, "entropy": r.entropy,
                "numbers": np.array([r.energy, r.expected_energy, r.prob, r.sign_energy, r.norm2])}
    if k == "sa":
        e, spins = ffi.sa_solve(probs, restarts=case["restarts"], sweeps=case["sweeps"], seed=state["seed"])
        return {"energy": e, "spins": np.concatenate(spins)}
    e, spins = learned.exact_ground(p)
    return {"energy": e, "spins": spins}


# ------------------------------------------------------------------------------------
# what one pass cannot do without
# ------------------------------------------------------------------------------------
def _updates(case, p):
    d = np.abs(p.ej - p.ei)
    return int((2 * d - 1).sum())


def _update_work(dl, dm, dr, keep, size):
    """Bytes and flops of one two-site update: contraction, thin SVD by bidiagonalisation with its
    left vectors (16 min(R, N) R N complex-counted flops), and the two new sites."""
    r, c = 2 * dl, 2 * dr
    return (size * (r * dm + dm * c + r * keep + keep * c),
            8.0 * r * dm * c + 16.0 * r * c * min(r, c) + 8.0 * keep * r * c)


def work(case):
    k = case["kind"]
    if k == "svd":
        r, c = case["rows"], case["cols"]
        m = min(r, c)
        return {"bytes": 16.0 * (r * c + m * (r + c)) + 8 * m, "flops": 24.0 * r * c * m}
    probs = _problems(case, 1)
    if k == "gnn":
        nodes, edges, h = sum(p.n for p in probs), 2 * sum(p.m for p in probs), case["hidden"]
        par = len(_gnn_params(case, np.random.Generator(np.random.PCG64(1))))
        mac = case["layers"] * (edges * h * (h + 1) + nodes * 2 * h * h) + 5 * nodes * h + case["count"] * h * h
        return {"bytes": 30.0 * par + 16.0 * nodes + 12.0 * edges, "flops": 6.0 * mac}
    if k in ("anneal", "batch"):
        size, by, fl = 16 if case["precision"] == "c128" else 8, 0.0, 0.0
        for p in probs:
            cap = min(case["chi"], 2 ** (p.n // 2)) / 2  # bonds fill up over the run
            b, f = _update_work(cap, cap, cap, cap, size)
            by += size * p.n * 2 * cap * cap
            fl += f * _updates(case, p) * case.get("stop", case["steps"])
        return {"bytes": by, "flops": fl}
    if k == "gates":
        chi, size = case["chi"], 16 if case["precision"] == "c128" else 8
        b, f = _update_work(chi, chi, chi, chi, size)
        return {"bytes": b * case["slots"] * case["count"], "flops": f * case["slots"] * case["count"]}
    if k == "sv":
        dim = 2.0 ** case["n"]
        return {"bytes": 40.0 * dim * case["steps"], "flops": (14.0 * case["n"] + 30.0) * dim * case["steps"]}
    if k == "sa":
        deg = sum(2 * p.m for p in probs)
        return {"bytes": 12.0 * deg, "flops": float(case["restarts"] * case["sweeps"]) * (deg + 20 * case["n"] * case["count"])}
    return {"bytes": 16.0 * probs[0].m + 8.0 * case["n"], "flops": 2.0 ** case["n"] * (case["n"] + 4.0)}


# ------------------------------------------------------------------------------------
# the same in 64 bits, without the framework
# ------------------------------------------------------------------------------------
def _slots(n, ei, ej):
    """Two-site slots (bond, edge or None for a swap) of one ZZ block, through the swap network."""
    out = []
    for e, (i, j) in enumerate(zip(ei, ej)):
        out += [(k - 1, None) for k in range(j, i + 1, -1)] + [(i, e)] + [(k, None) for k in range(i + 1, j)]
    return out


def _two_site(sites, bond, gate, chi):
    """One update with numpy's SVD: keep at most chi values, none below rounding; returns the
    discarded weight's share."""
    a, c = sites[bond], sites[bond + 1]
    dl, dr = a.shape[0], c.shape[2]
    t = np.tensordot(a, c, (2, 0))
    if gate is None:
        t = t.transpose(0, 2, 1, 3)
    else:
        t = t * np.array([[gate, gate.conjugate()], [gate.conjugate(), gate]])[None, :, :, None]
    th = t.reshape(2 * dl, 2 * dr)
    u, s, vh = np.linalg.svd(th, full_matrices=False)
    floor = max(1e-14, 8.0 * math.sqrt(2 * dl) * 2.0 ** -52 * float(np.linalg.norm(s)))
    keep = max(1, int((s[:chi] >= floor).sum()))
    sites[bond] = u[:, :keep].reshape(dl, 2, keep)
    sites[bond + 1] = (u[:, :keep].conj().T @ th).reshape(keep, 2, dr)
    return float((s[keep:] ** 2).sum() / (s ** 2).sum())


def _one_site(p, k, i):
    nx, nz = -p.sa[k], -p.sb[k] * p.h[i]
    r = math.hypot(nx, nz)
    c, s = (math.cos(0.5 * p.dt * r), math.sin(0.5 * p.dt * r) / r) if r > 0 else (1.0, 0.0)
    return np.array([[c - 1j * s * nz, -1j * s * nx], [-1j * s * nx, c + 1j * s * nz]])


def _entropy0(sites):
    e = np.ones((1, 1), np.complex128)
    for t in reversed(sites[1:]):
        e = np.einsum("asx,bsx->ab", np.tensordot(t, e, (2, 0)), t.conj())
    rho = np.einsum("sx,xy,ty->st", sites[0][0], e, sites[0][0].conj())
    lam = np.clip(np.linalg.eigvalsh(rho / np.trace(rho).real), 0.0, 1.0)
    return -sum(x * math.log2(x) for x in lam if x > 1e-12)


def _signs(n):
    x = np.arange(1 << n)
    return [1.0 - 2.0 * ((x >> i) & 1) for i in range(n)]


def _energies(p, z):
    e = np.zeros_like(z[0])
    for i, j, w in zip(p.ei, p.ej, p.ew):
        e -= w * z[i] * z[j]
    for i in range(p.n):
        e -= p.h[i] * z[i]
    return e


def _readout(p, psi):
    """(spins, energy, <H>, probability of the spins, norm, <Z>) of a dense state."""
    z = _signs(p.n)
    pr = np.abs(psi) ** 2
    nrm = pr.sum()
    ez = np.array([(pr * zi).sum() / nrm for zi in z])
    spins = np.where(ez >= 0, 1, -1).astype(np.int8)
    en = _energies(p, z)
    x = int(sum(1 << i for i in range(p.n) if spins[i] < 0))
    return spins, en[x], (pr * en).sum() / nrm, pr[x] / nrm, nrm, ez


def _dense_host(sites):
    v = np.ones((1, 1), np.complex128)
    for t in sites:
        w = (v @ t.reshape(t.shape[0], -1)).reshape(v.shape[0], 2, t.shape[2])
        v = w.transpose(1, 0, 2).reshape(-1, t.shape[2])
    return v[:, 0]


def _exact_anneal(p, chi, stop):
    sites = [np.full((1, 2, 1), math.sqrt(0.5), np.complex128) for _ in range(p.n)]
    ent, worst = [], 0.0
    slots = _slots(p.n, p.ei, p.ej)
    for k in range(stop):
        g = [_one_site(p, k, i) for i in range(p.n)]
        for half in (0, 1):
            sites = [np.einsum("st,atb->asb", g[i], t) for i, t in enumerate(sites)]
            if half == 0:
                for bond, e in slots:
                    gate = None if e is None else np.exp(1j * p.dt * p.sb[k] * p.ew[e])
                    worst = max(worst, _two_site(sites, bond, gate, chi))
        ent.append(_entropy0(sites))
    return _readout(p, _dense_host(sites)), np.array(ent), worst


def _exact_dense(p, chi):
    """The same anneal at bonds that never truncate: the dense state, step by step."""
    n = p.n
    z = _signs(n)
    zz = np.zeros(1 << n)
    for i, j, w in zip(p.ei, p.ej, p.ew):
        zz -= w * z[i] * z[j]
    psi = np.full(1 << n, 2.0 ** (-0.5 * n), np.complex128)
    ent = []
    for k in range(p.steps):
        for half in (0, 1):
            for i in range(n):
                psi = np.einsum("st,atb->asb", _one_site(p, k, i), psi.reshape(-1, 2, 1 << i)).reshape(-1)
            if half == 0:
                psi = psi * np.exp(-1j * p.dt * p.sb[k] * zz)
        m = psi.reshape(-1, 2)
        rho = m.T @ m.conj()
        lam = np.clip(np.linalg.eigvalsh(rho / np.trace(rho).real), 0.0, 1.0)
        ent.append(-sum(x * math.log2(x) for x in lam if x > 1e-12))
    return _readout(p, psi), np.array(ent), 0.0


def _random_mps(n, cap, seed, decay):
    """The random MPS of `Session.randomize`: complex normal entries from splitmix64, column b of
    every site scaled by exp(-b / decay)."""
    dims = [min(cap, 2 ** i, 2 ** (n - i)) for i in range(n + 1)]
    sites = []
    with np.errstate(over="ignore"):
        for i in range(n):
            dl, dr = dims[i], dims[i + 1]
            t = np.arange(dl * 2 * dr, dtype=np.uint64)
            z = np.uint64(seed) ^ np.uint64(i << 40) ^ (t * np.uint64(0x9E3779B97F4A7C15))
            u = []
            for _ in range(2):
                z = z + np.uint64(0x9E3779B97F4A7C15)
                x = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
                x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
                u.append((x ^ (x >> np.uint64(31))) >> np.uint64(11))
            r = np.sqrt(-2.0 * np.log((u[0].astype(np.float64) + 0.5) * 2.0 ** -53)) / math.sqrt(2.0 * dl)
            r = r * np.exp(-(t % np.uint64(dr)).astype(np.float64) / decay)
            sites.append((r * np.exp(2j * math.pi * u[1].astype(np.float64) * 2.0 ** -53)).reshape(dl, 2, dr))
    return sites


def _exact_gates(case, p, seed):
    sites = _random_mps(case["n"], case["chi"], seed, case["decay"])
    if case["precision"] == "c64":
        sites = [t.astype(np.complex64).astype(np.complex128) for t in sites]
    first, last = _window(case)
    worst = 0.0
    for bond, e in _slots(p.n, p.ei, p.ej)[first:last]:
        gate = None if e is None else np.exp(1j * p.dt * p.sb[20] * p.ew[e])
        worst = max(worst, _two_site(sites, bond, gate, case["chi"]))
    return sites, worst


def _exact_sv(p, mode):
    """The state-vector anneal in torch, complex128 on the GPU."""
    n, dev = p.n, "cuda"
    x = torch.arange(1 << n, device=dev)
    z = [(1 - 2 * ((x >> i) & 1)).double() for i in range(n)]
    zz = torch.zeros(1 << n, dtype=torch.float64, device=dev)
    for i, j, w in zip(p.ei.tolist(), p.ej.tolist(), p.ew.tolist()):
        zz -= w * z[i] * z[j]
    en = zz.clone()
    for i in range(n):
        en -= float(p.h[i]) * z[i]
    psi = torch.full((1 << n,), 2.0 ** (-0.5 * n), dtype=torch.complex128, device=dev)

    def gates(k, f):
        nonlocal psi
        for i in range(n):
            g = torch.from_numpy(f(k, i)).to(dev)
            v = psi.reshape(-1, 2, 1 << i)
            a, b = v[:, 0], v[:, 1]
            psi = torch.stack([g[0, 0] * a + g[0, 1] * b, g[1, 0] * a + g[1, 1] * b], 1).reshape(-1)

    ent = []
    for k in range(p.steps):
        if mode == 0:
            ph = torch.exp(-0.5j * p.dt * float(p.sb[k]) * en)
            psi = psi * ph
            c, s = math.cos(p.sa[k] * p.dt), math.sin(p.sa[k] * p.dt)
            gates(k, lambda k, i: np.array([[c, 1j * s], [1j * s, c]]))
            psi = psi * ph
        else:
            gates(k, lambda k, i: _one_site(p, k, i))
            psi = psi * torch.exp(-1j * p.dt * float(p.sb[k]) * zz)
            gates(k, lambda k, i: _one_site(p, k, i))
        m = psi.reshape(-1, 2)
        rho = (m.T @ m.conj()).cpu().numpy()
        lam = np.clip(np.linalg.eigvalsh(rho / np.trace(rho).real), 0.0, 1.0)
        ent.append(-sum(v * math.log2(v) for v in lam if v > 1e-12))
    pr = psi.abs() ** 2
    nrm = float(pr.sum())
    best = int(pr.argmax())
    ez = np.array([float((pr * zi).sum()) for zi in z])
    xs = int(sum(1 << i for i in range(n) if ez[i] < 0))
    return {"entropy": np.array(ent),
            "numbers": np.array([float(en[best]), float((pr * en).sum()) / nrm, float(pr[best]) / nrm,
                                 float(en[xs]), nrm])}


def _gnn_shapes(case):
    h, k = case["hidden"], case["knots"]
    out = [("We", (h, 4)), ("be", (h,))]
    for l in range(case["layers"]):
        out += [("W1%d" % l, (h, h + 1)), ("b1%d" % l, (h,)), ("W2%d" % l, (h, 2 * h)), ("b2%d" % l, (h,))]
    return out + [("wn", (h,)), ("bn", (1,)), ("Wg1", (h, h)), ("bg1", (h,)), ("Wg2", (k - 1, h)), ("bg2", (k - 1,))]


def _gnn_params(case, rng):
    """Weights uniform over the fan-in, small enough that no spin's probability saturates."""
    out = []
    for name, shape in _gnn_shapes(case):
        fan = shape[-1] if len(shape) > 1 or name == "wn" else 0
        scale = 0.1 if name == "Wg2" else 0.3 if name[:2] in ("W1", "W2", "wn") else 1.0
        a = scale * math.sqrt(6.0 / fan) if fan else 0.05
        out.append(rng.uniform(-a, a, int(np.prod(shape))))
    return np.concatenate(out).astype(np.float32)


def _exact_gnn(case, seed):
    probs, knots, spins, params = _gnn_inputs(case, seed)
    flat = torch.from_numpy(params).to(torch.bfloat16).double().requires_grad_()
    w, o = {}, 0
    for name, shape in _gnn_shapes(case):
        m = int(np.prod(shape))
        w[name] = flat[o:o + m].reshape(shape)
        o += m
    feat, src, dst, ew, goff = [], [], [], [], [0]
    for p in probs:
        sa, ss, j = np.zeros(p.n), np.zeros(p.n), p.ew.astype(np.float32).astype(np.float64)
        for a, b in ((p.ei, p.ej), (p.ej, p.ei)):
            np.add.at(sa, a, np.abs(j))
            np.add.at(ss, a, j)
            src.append(a + goff[-1])
            dst.append(b + goff[-1])
            ew.append(j)
        feat.append(np.stack([p.h, sa / 4, ss / 4, np.ones(p.n)], 1))
        goff.append(goff[-1] + p.n)
    src, dst = torch.from_numpy(np.concatenate(src)), torch.from_numpy(np.concatenate(dst))
    ew = torch.from_numpy(np.concatenate(ew))[:, None]
    x = torch.relu(torch.from_numpy(np.concatenate(feat)) @ w["We"].T + w["be"])
    for l in range(case["layers"]):
        m = torch.relu(torch.cat([x[src], ew], 1) @ w["W1%d" % l].T + w["b1%d" % l])
        a = torch.zeros_like(x).index_add(0, dst, m)
        x = x + torch.relu(torch.cat([x, a], 1) @ w["W2%d" % l].T + w["b2%d" % l])
    t = torch.from_numpy(spins).double()
    loss = 0.2 * torch.nn.functional.binary_cross_entropy_with_logits(x @ w["wn"] + w["bn"], t)
    g = torch.stack([x[a:b].mean(0) for a, b in zip(goff, goff[1:])])
    d = torch.nn.functional.softplus(torch.relu(g @ w["Wg1"].T + w["bg1"]) @ w["Wg2"].T + w["bg2"])
    c = torch.cat([torch.zeros(len(probs), 1, dtype=torch.float64), d.cumsum(1)], 1)
    loss = loss + ((c / c[:, -1:] - torch.from_numpy(knots).double()) ** 2).mean()
    loss.backward()
    return {"loss": np.array([loss.item()], np.float64), "grads": flat.grad.numpy()}


def exact(case, seed):
    k = case["kind"]
    if k == "svd":
        u, s, vh = np.linalg.svd(_matrix(case, seed), full_matrices=False)
        ph = u[0] / np.abs(u[0])
        return {"u": u * ph.conj(), "s": s, "vh": vh * ph[:, None]}
    if k == "gnn":
        return _exact_gnn(case, seed)
    probs = _problems(case, seed)
    p = probs[0]
    if k == "anneal":
        (spins, e, eh, pr, nrm, ez), ent, worst = _exact_anneal(p, case["chi"], case["stop"])
        if case["legacy"]:
            return {"spins": None, "energy": float(e), "entropy": ent}
        return {"spins": None, "numbers": np.append([e, eh, pr, nrm, worst], ez), "entropy": ent}
    if k == "batch":
        if any(2 ** (q.n // 2) > case["chi"] for q in probs):
            return None  # truncating: some ten thousand SVDs
        r = [_exact_dense(q, case["chi"]) for q in probs]
        return {"spins": None, "numbers": np.concatenate([np.append([*x[0][1:5], x[2]], x[0][5]) for x in r]),
                "entropy": np.concatenate([x[1] for x in r])}
    if k == "gates":
        worst = []
        out = {}
        for b in sorted({0, case["count"] - 1}):
            sites, w = _exact_gates(case, probs[b], seed + 7919 * b)
            out["state%d" % (b > 0)] = psi = _dense_host(sites)
            worst.append(w)
        if case["count"] > 1:
            return {"kept": None, **out}  # the largest discarded weight is over all instances
        _, e, eh, pr, nrm, _ = _readout(p, psi)
        return {"kept": np.array([1.0 - worst[0]]), "spins": None, "numbers": np.array([e, eh, pr, nrm]), **out}
    if k == "sv":
        return _exact_sv(p, case["mode"])
    if k == "sa":
        return None  # a search: its answer is the draws' own
    n = p.n
    best = math.inf
    for c in range(0, 1 << n, 1 << 20):
        x = np.arange(c, min(c + (1 << 20), 1 << n))
        z = [2.0 * ((x >> i) & 1) - 1.0 for i in range(n)]
        best = min(best, float(_energies(p, z).min()))
    return {"energy": best, "spins": None}
