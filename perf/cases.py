"""The work that programs have this package do, as cases to be timed: Krylov time steps from the
smallest register to the largest, a whole run of the time loop, H*psi, a measurement of the
observables, gradients of a step and of whole pulses, a batch of registers, the noisy state-vector
step and the density-matrix step.

A case is a dict of plain values.  ``prepare`` makes its inputs from the case and a seed, ``run``
is one pass through the public entry points, ``exact`` the same outputs in complex128 by plain
torch (a Chebyshev expansion of the exponential).

Units follow the steppers: rad/us, us and um; ``U_ij = C6 / r_ij**6``.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

C6 = 5420158.53
TOL = 1e-10
DEV = "cuda"


# ------------------------------------------------------------------------------- cases
def listed():
    return [
        # one time step of the N=10 chain (5 um, dt = 10 ns): the smallest calls, all latency
        {"name": "step_n10_c128", "kind": "step", "n": 10, "register": "chain", "dtype": "c128",
         "dt": 0.01, "phase": False},
        # a whole short sequence through the backend: 20 steps of a 12-atom ladder with
        # occupation, correlation and energy read four times
        {"name": "run_n12_c128", "kind": "run", "n": 12, "register": "ladder", "dtype": "c128",
         "dt": 0.01, "phase": False, "steps": 20, "every": 5},
        # a step of an irregular register with laser phases, in the single-precision form
        {"name": "step_n15_c64", "kind": "step", "n": 15, "register": "box", "dtype": "c64",
         "dt": 0.01, "phase": True},
        # a step of the N=20 4x5 lattice (6 um, dt = 10 ns), complex128
        {"name": "step_n20_c128", "kind": "step", "n": 20, "register": "lattice", "dtype": "c128",
         "dt": 0.01, "phase": False},
        # a step of the N=26 2x13 ladder (5.5 um, dt = 5 ns), complex64: the largest register
        {"name": "step_n26_c64", "kind": "step", "n": 26, "register": "ladder", "dtype": "c64",
         "dt": 0.005, "phase": False},
        # the operator by itself, as programs that bring their own propagator use it
        {"name": "hpsi_n23_c128", "kind": "hpsi", "n": 23, "register": "box", "dtype": "c128",
         "dt": 0.01, "phase": True},
        # every observable of a large state: occupation, correlation matrix, 1000 bitstrings,
        # and of a complex128 state the energy and its variance
        {"name": "observe_n22_c128", "kind": "observe", "n": 22, "register": "box", "dtype": "c128",
         "dt": 0.01, "phase": False, "shots": 1000},
        # one differentiable step, forward and backward, with the gradients of the pulse, the
        # interactions and the state
        {"name": "grad_n13_c128", "kind": "grad", "n": 13, "register": "box", "dtype": "c128",
         "dt": 0.01, "phase": True},
        # pulse optimisation: the gradients of several parameter sets of a ring (20-ns-and-up
        # segments, Neel target), forward and adjoint over all steps
        {"name": "pulse_n14_c128", "kind": "pulse", "n": 14, "register": "ring", "dtype": "c128",
         "dt": 0.01, "phase": False, "sets": 12, "segments": 2, "steps": 5},
        # many registers of uneven size evolved together, complex64
        {"name": "batch_40_c64", "kind": "batch", "n": 12, "nmax": 18, "dtype": "c64", "dt": 0.01,
         "registers": 40, "steps": 30, "phase": False},
        # a Monte Carlo trajectory's step with a jump: the noisy exponential, the jump weights
        # of every qubit and operator, the operator applied
        {"name": "jump_n19_c128", "kind": "jump", "n": 19, "register": "box", "dtype": "c128",
         "dt": 0.01, "phase": False},
        # a step of a density matrix under relaxation and dephasing (2^20 entries)
        {"name": "lindblad_n10_c128", "kind": "lindblad", "n": 10, "register": "ladder",
         "dtype": "c128", "dt": 0.01, "phase": False},
    ]


def draw(rng):
    """One more case of the same ranges (qubit numbers are the logarithm of the sizes).  Whole
    runs, gradients and trajectories are drawn in complex128, the precision they default to."""
    kind = rng.choice(["step", "step", "step", "run", "hpsi", "observe", "grad", "pulse", "batch",
                       "jump", "lindblad"])
    c = {"kind": kind, "dtype": rng.choice(["c64", "c128"]), "dt": rng.choice([0.004, 0.005, 0.008, 0.01]),
         "phase": rng.random() < 0.4}
    if kind in ("run", "grad", "pulse", "jump"):
        c["dtype"] = "c128"
    reg = rng.choice(["chain", "ladder", "box", "box"])
    if kind == "step":
        c |= {"n": rng.randint(7, 24), "register": reg}
    elif kind == "run":
        c |= {"n": rng.randint(8, 16), "register": reg, "steps": rng.randint(6, 24), "every": rng.randint(2, 6)}
    elif kind == "hpsi":
        c |= {"n": rng.randint(10, 24), "register": reg}
    elif kind == "observe":
        c |= {"n": rng.randint(10, 24), "register": reg, "shots": rng.randint(100, 3000)}
    elif kind == "grad":
        c |= {"n": rng.randint(8, 16), "register": reg}
    elif kind == "pulse":
        c |= {"n": rng.randint(9, 14), "register": "ring", "phase": False, "sets": rng.randint(2, 12),
              "segments": rng.randint(2, 3), "steps": rng.randint(2, 4)}
    elif kind == "batch":
        n = rng.randint(9, 13)
        c |= {"n": n, "nmax": n + rng.randint(1, 4), "registers": rng.randint(5, 40), "steps": rng.randint(5, 24)}
    elif kind == "jump":
        c |= {"n": rng.randint(8, 20), "register": reg}
    else:
        c |= {"n": rng.randint(3, 10), "register": reg}
    return c


# ------------------------------------------------------------------------------ inputs
def _dtype(c):
    return torch.complex64 if c["dtype"] == "c64" else torch.complex128


def _positions(kind, n, rng):
    if kind == "chain":
        return np.stack([5.0 * np.arange(n), np.zeros(n)], 1)
    if kind == "ladder":
        k = np.arange(n)
        return 5.5 * np.stack([k // 2, k % 2], 1).astype(float)
    if kind == "lattice":
        k = np.arange(n)
        return 6.0 * np.stack([k % 5, k // 5], 1).astype(float)
    if kind == "ring":
        a = 2.0 * np.pi * np.arange(n) / n
        return 10.0 * np.stack([np.cos(a), np.sin(a)], 1)
    pts = []  # uniform in a 40 x 40 um box, at least 5 um apart
    while len(pts) < n:
        p = rng.uniform(0.0, 40.0, 2)
        if all(np.hypot(*(p - q)) >= 5.0 for q in pts):
            pts.append(p)
    return np.array(pts)


def _interactions(pos):
    d = pos[:, None] - pos[None]
    r2 = (d * d).sum(-1)
    np.fill_diagonal(r2, np.inf)
    return C6 / r2 ** 3


def _diagonal(de, U, n):
    """-sum_i delta_i n_i + sum_{i<j} U_ij n_i n_j over the 2^n bitstrings, float64 on the GPU."""
    d = torch.zeros(1 << n, dtype=torch.float64, device=DEV)
    for i in range(n):
        v = d.view(1 << i, 2, -1)
        v[:, 1] -= float(de[i])
        for j in range(i + 1, n):
            d.view(1 << i, 2, 1 << (j - i - 1), 2, -1)[:, 1, :, 1] += float(U[i, j])
    return d


def _evolved(om, de, U, n, dtype, rng):
    """A state partway through a sequence: a few split steps of the drive from |g...g>."""
    steps, h = 6, 0.03
    ph = torch.exp(-1j * h * _diagonal(de, U, n)).to(dtype)
    psi = torch.zeros(1 << n, dtype=dtype, device=DEV)
    psi[0] = 1.0
    for _ in range(steps):
        for i in range(n):
            a = 0.5 * h * float(om[i]) * rng.uniform(0.8, 1.2)
            v = psi.view(1 << i, 2, -1)
            psi = (math.cos(a) * v - 1j * math.sin(a) * v.flip(1)).reshape(-1)
        psi = psi * ph
    return (psi / torch.linalg.vector_norm(psi)).to(dtype)


def _drive(c, rng):
    """Omega, delta, phi of one step and U, float64 on the host, as the sequence adapter gives them."""
    n = c["n"]
    U = _interactions(_positions(c["register"], n, rng))
    om = np.full(n, rng.uniform(3.0, 6.0))
    de = np.full(n, rng.uniform(-8.0, 8.0))
    ph = rng.uniform(0.0, 2.0 * np.pi, n) if c["phase"] else np.zeros(n)
    return [torch.as_tensor(a) for a in (om, de, ph, U)]


def _random_like(psi, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randn(psi.numel(), 2, dtype=torch.float64, device=DEV, generator=g)
    return (torch.view_as_complex(w) / math.sqrt(2.0 * psi.numel())).to(psi.dtype)


def _lindblads():
    c = math.sqrt(0.5)
    return [torch.tensor([[0.0, c], [0.0, 0.0]], dtype=torch.complex128),
            torch.tensor([[c, 0.0], [0.0, -c]], dtype=torch.complex128)]


def _inputs(c, seed):
    """What the case's call is given, as plain tensors and arrays."""
    rng = np.random.default_rng(seed)
    k, n = c["kind"], c["n"]
    if k == "pulse":
        U = _interactions(_positions("ring", n, rng))
        return {"U": U, "om": rng.uniform(0.0, 2.0 * np.pi, (c["sets"], c["segments"])),
                "de": rng.uniform(-20.0, 20.0, (c["sets"], c["segments"])),
                "target": (np.arange(n) + 1.0) % 2}
    t = (np.arange(c.get("steps", 1)) + 0.5) / c.get("steps", 1)
    if k == "batch":
        sizes, regs = np.linspace(n, c["nmax"] + 0.99, c["registers"]).astype(int), []
        kt = np.linspace(0.0, 1.0, 11)
        for m in sizes:
            om = np.interp(t, kt, rng.uniform(0.0, 2.0 * np.pi, 11))
            de = np.interp(t, kt, rng.uniform(-20.0, 20.0, 11))
            ph = rng.uniform(0.0, 2.0 * np.pi, m) if c["phase"] else np.zeros(m)
            wide = np.ones((1, m))
            regs.append((_interactions(_positions("box", m, rng)), om[:, None] * wide,
                         de[:, None] * wide, np.ones((len(t), 1)) * ph))
        return {"registers": regs}
    om, de, ph, U = _drive(c, rng)
    if k == "run":
        wide = torch.ones(c["steps"], 1, dtype=torch.float64)
        return {"om": om * wide, "de": torch.as_tensor(-10.0 + 20.0 * t)[:, None] + de * wide * 0.1,
                "ph": ph * wide, "U": U}
    psi = _evolved(om, de, U, n, _dtype(c), rng)
    s = {"om": om, "de": de, "ph": ph, "U": U, "psi": psi}
    if k == "grad":
        s["w"] = _random_like(psi, seed)
    if k == "observe":
        s["u"] = torch.as_tensor(rng.random(c["shots"]), device=DEV)
    if k == "lindblad":
        other = _evolved(0.7 * om, de, U, n, _dtype(c), rng)
        s["rho"] = 0.8 * torch.outer(psi, psi.conj()) + 0.2 * torch.outer(other, other.conj())
        del s["psi"]
    return s


class _Register:
    """One register of a batch, with the attributes BatchEvolution reads."""

    def __init__(self, U, omega, delta, phi, dt):
        self.U, self.omega, self.delta, self.phi, self.dt, self.tolerance = U, omega, delta, phi, dt, TOL


# --------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    from emulators_b200 import EvolveMonteCarlo, EvolveStateVector, RydbergHamiltonian
    from emulators_b200.batch import BatchEvolution
    from emulators_b200.gradients import PulseGradientBatch
    from emulators_b200.sv_backend import (CorrelationMatrix, Energy, Occupation, SequenceData, StateResult,
                                           SVConfig)
    from emulators_b200.time_evolution import EvolveDensityMatrix

    s = _inputs(case, seed)
    s["case"] = case
    k = case["kind"]
    if k in ("step", "grad"):
        s["stepper"] = EvolveStateVector(100)
    elif k == "run":
        nst = case["steps"]
        at = [e / nst for e in range(case["every"], nst + 1, case["every"])]
        s["data"] = SequenceData(s["om"], s["de"], s["ph"], [1000.0 * case["dt"] * j for j in range(nst + 1)], s["U"])
        s["config"] = SVConfig(dt=1000.0 * case["dt"], krylov_tolerance=TOL, precision=case["dtype"],
                               observables=[Occupation(at), CorrelationMatrix(at), Energy(at),
                                            StateResult([1.0])])
    elif k in ("hpsi", "observe"):
        s["H"] = RydbergHamiltonian(s["om"], s["de"], s["ph"], s["U"], DEV)
    elif k == "pulse":
        s["batch"] = PulseGradientBatch(s["U"], case["dt"], s["om"], s["de"], case["steps"], s["target"],
                                        precision=case["dtype"], tolerance=TOL, max_krylov_dim=120)
    elif k == "batch":
        s["batch"] = BatchEvolution([_Register(*r, case["dt"]) for r in s["registers"]], case["dtype"])
    elif k == "jump":
        s["stepper"] = EvolveMonteCarlo(100)
        s["ops"] = _lindblads()
        st = torch.stack(s["ops"])
        s["weights"] = st.conj().transpose(1, 2) @ st
    elif k == "lindblad":
        s["stepper"] = EvolveDensityMatrix(100)
        s["ops"] = _lindblads()
    return s


def run(s):
    from emulators_b200 import (StateVector, apply, correlation_matrix_sv_impl, energy_sv_impl,
                                energy_variance_sv_impl, expect_batch, qubit_occupation_sv_impl)
    from emulators_b200.state_vector import sample_indices
    from emulators_b200.sv_backend import SVBackend

    case = s["case"]
    k, dt = case["kind"], case["dt"]
    if k == "step":
        return s["stepper"].apply(dt, s["om"], s["de"], s["ph"], s["U"], s["psi"], TOL, None)[0]
    if k == "run":
        r = SVBackend(s["data"], s["config"]).run()
        return [*(torch.stack(r.get(t)) for t in ("occupation", "correlation_matrix", "energy")),
                r.get("state")[0].data]
    if k == "hpsi":
        return s["H"] * s["psi"]
    if k == "observe":
        st, H = StateVector(s["psi"]), s["H"]
        out = [qubit_occupation_sv_impl(state=st), correlation_matrix_sv_impl(state=st),
               sample_indices(s["psi"], s["u"])]
        if case["dtype"] == "c128":
            out += [energy_sv_impl(state=st, hamiltonian=H), energy_variance_sv_impl(state=st, hamiltonian=H)]
        return out
    if k == "grad":
        x = [s[q].detach().requires_grad_() for q in ("om", "de", "ph", "U", "psi")]
        out = s["stepper"].apply(dt, *x, TOL, None)[0]
        return [out.detach(), *torch.autograd.grad(out, x, s["w"])]
    if k == "pulse":
        return list(s["batch"].loss_and_grad())
    if k == "batch":
        s["batch"].run()
        return s["batch"].states
    if k == "jump":
        ham = s["stepper"].get_hamiltonian(s["om"], s["de"], s["ph"], s["ops"], s["U"], DEV)
        psi = s["stepper"].evolve(dt, ham, s["psi"], TOL)
        w = expect_batch(psi, s["weights"], case["n"])
        return [psi, w, apply(psi, case["n"] // 2, s["ops"][0])]
    return s["stepper"].apply(dt, s["om"], s["de"], s["ph"], s["U"], s["rho"], TOL, s["ops"])[0]


def work(case):
    """One pass's bytes and operations: a Krylov step of m iterations over D amplitudes of s bytes
    reads and writes (7 m + 1) D s and takes about m D (8 n + 40) operations; m is a nominal count."""
    n, k = case["n"], case["kind"]
    size, D = (8 if case["dtype"] == "c64" else 16), float(1 << n)

    def steps(m, amps, qubits, count=1.0):
        return {"bytes": count * (7 * m + 1) * amps * size, "flops": count * m * amps * (8 * qubits + 40)}

    if k == "hpsi":
        return {"bytes": 2 * D * size, "flops": D * (8 * n + 8)}
    if k == "observe":
        return {"bytes": 4 * D * size, "flops": D * (8 * n + 40)}
    if k == "step":
        return steps(20, D, n)
    if k == "run":
        return steps(20, D, n, case["steps"])
    if k == "grad":
        return steps(20, D, n, 4)
    if k == "pulse":
        return steps(50, D, n, 4.0 * case["sets"] * case["segments"] * case["steps"])
    if k == "batch":
        ns = np.linspace(n, case["nmax"] + 0.99, case["registers"]).astype(int)
        return steps(20, float((2.0 ** ns).sum()), n, case["steps"])
    if k == "jump":  # Arnoldi: every iteration reads the whole basis
        return {"bytes": 20 * 26 * D * size, "flops": 20 * D * (8 * n + 8 * 20)}
    return {"bytes": 20 * 26 * D * D * size, "flops": 20 * D * D * (16 * n + 8 * 20)}


# ------------------------------------------------------------------------------- exact
def _expm(apply_h, lo, hi, dt, v):
    """exp(-i dt H) v for H = apply_h with its real spectrum in [lo, hi], by the Chebyshev
    expansion (coefficients by a cosine transform of the exponential on the interval)."""
    mid, half = 0.5 * (lo + hi), max(0.5 * (hi - lo), 1e-9)
    z = dt * half
    M = 4 * int(2.0 * abs(z) + 64)
    th = np.pi * (np.arange(M) + 0.5) / M
    K = int(1.2 * abs(z) + 50)
    f = np.exp(-1j * z * np.cos(th))
    coef = [(2.0 - (k == 0)) / M * (f * np.cos(k * th)).sum() * np.exp(-1j * dt * mid) for k in range(K)]
    a, b = v, (apply_h(v) - mid * v) / half
    out = complex(coef[0]) * a + complex(coef[1]) * b
    for k in range(2, K):
        a, b = b, (2.0 / half) * (apply_h(b) - mid * b) - a
        out = out + complex(coef[k]) * b
    return out


def _xor_index(n):
    x = torch.arange(1 << n, device=DEV)
    return torch.stack([x ^ (1 << (n - 1 - i)) for i in range(n)])


def _operator(om, de, ph, U, n, noise=None, idx=None):
    """(psi -> H psi, lowest, highest energy bound): gathered flips on small registers."""
    om, de, ph, U = (a.detach().cpu().double().numpy() if isinstance(a, torch.Tensor) else np.asarray(a)
                     for a in (om, de, ph, U))
    d = _diagonal(de, U, n)
    up = 0.5 * om * np.exp(1j * ph)
    dn = up.conj()
    span = np.abs(up).sum() + 1e-3
    if noise is not None:
        up, dn = up + complex(noise[1, 0]), dn + complex(noise[0, 1])
        pop = _diagonal(-np.ones(n), np.zeros((n, n)), n)
        d = d + n * complex(noise[0, 0]) + pop * (complex(noise[1, 1]) - complex(noise[0, 0]))
    lo, hi = float(d.real.min()) - span, float(d.real.max()) + span
    if n <= 18:
        idx = _xor_index(n) if idx is None else idx
        bit = (torch.arange(1 << n, device=DEV)[None] >> torch.arange(n - 1, -1, -1, device=DEV)[:, None]) & 1
        if not np.any(up.imag) and not np.any(dn.imag) and noise is None:
            cf = torch.as_tensor(up.real, device=DEV)[:, None]
        else:
            u, w = (torch.as_tensor(a, device=DEV)[:, None] for a in (up, dn))
            cf = torch.where(bit == 1, u, w)
        return (lambda p: d * p + (cf * p[idx]).sum(0)), lo, hi

    def h(p):
        out = d * p
        for i in range(n):
            v, o = p.view(1 << i, 2, -1), out.view(1 << i, 2, -1)
            o[:, 1] += complex(up[i]) * v[:, 0]
            o[:, 0] += complex(dn[i]) * v[:, 1]
        return out

    return h, lo, hi


def _occupation(p2, n):
    return torch.stack([p2.view(1 << i, 2, -1)[:, 1].sum() for i in range(n)])


def _correlation(p2, n):
    out = torch.zeros(n, n, dtype=torch.float64)
    for i in range(n):
        out[i, i] = p2.view(1 << i, 2, -1)[:, 1].sum().cpu()
        for j in range(i + 1, n):
            out[i, j] = out[j, i] = p2.view(1 << i, 2, 1 << (j - i - 1), 2, -1)[:, 1, :, 1].sum().cpu()
    return out


def _noise():
    st = torch.stack(_lindblads())
    return (-0.5j * (st.conj().transpose(1, 2) @ st).sum(0)).numpy()


def exact(case, seed):
    s = _inputs(case, seed)
    k, n, dt = case["kind"], case["n"], case["dt"]
    if k == "pulse":
        return _exact_pulse(case, s)
    if k == "batch":
        return _exact_batch(case, s)
    if k == "grad":
        return _exact_grad(case, s)
    if k == "lindblad":
        return _exact_lindblad(case, s)
    if k == "run":
        psi = torch.zeros(1 << n, dtype=torch.complex128, device=DEV)
        psi[0] = 1.0
        occ, cor, en = [], [], []
        for j in range(case["steps"]):
            h, lo, hi = _operator(s["om"][j], s["de"][j], s["ph"][j], s["U"], n)
            psi = _expm(h, lo, hi, dt, psi)
            if (j + 1) % case["every"] == 0:
                p2 = psi.abs() ** 2
                occ.append(_occupation(p2, n))
                cor.append(_correlation(p2, n))
                en.append(torch.vdot(psi, h(psi)).real)
        return [torch.stack(occ), torch.stack(cor), torch.stack(en), psi]
    psi = s["psi"].to(torch.complex128)
    if k == "jump":
        ops = _lindblads()
        h, lo, hi = _operator(s["om"], s["de"], s["ph"], s["U"], n, _noise())
        psi = _expm(h, lo, hi, dt, psi)
        rho = torch.stack([torch.einsum("aib,ajb->ij", psi.view(1 << i, 2, -1), psi.view(1 << i, 2, -1).conj())
                           for i in range(n)])
        agg = torch.stack([L.conj().T @ L for L in ops]).to(DEV)
        v = psi.view(1 << (n // 2), 2, -1)
        return [psi, torch.einsum("kab,qba->qk", agg, rho),
                torch.einsum("ij,ajb->aib", ops[0].to(DEV), v).reshape(-1)]
    h, lo, hi = _operator(s["om"], s["de"], s["ph"], s["U"], n)
    if k == "step":
        return _expm(h, lo, hi, dt, psi)
    if k == "hpsi":
        return h(psi)
    hp, p2 = h(psi), psi.abs() ** 2
    e = torch.vdot(psi, hp).real
    out = [_occupation(p2, n), _correlation(p2, n), None]
    return out + [e, torch.vdot(hp, hp).real - e ** 2] if case["dtype"] == "c128" else out


def _exact_batch(case, s):
    out, index = [], {}
    for U, om, de, ph in s["registers"]:
        n = U.shape[0]
        index.setdefault(n, _xor_index(n))
        psi = torch.zeros(1 << n, dtype=torch.complex128, device=DEV)
        psi[0] = 1.0
        for j in range(case["steps"]):
            psi = _expm(*_operator(om[j], de[j], ph[j], U, n, idx=index[n]), case["dt"], psi)
        out.append(psi)
    return torch.cat(out)


def _exact_grad(case, s):
    n, dt = case["n"], case["dt"]
    _, lo, hi = _operator(s["om"], s["de"], s["ph"], s["U"], n)
    x = [s[q].to(DEV, torch.float64).requires_grad_() for q in ("om", "de", "ph", "U")]
    psi = s["psi"].to(torch.complex128).requires_grad_()
    om, de, ph, U = x
    idx = _xor_index(n)
    bit = ((torch.arange(1 << n, device=DEV)[None] >> torch.arange(n - 1, -1, -1, device=DEV)[:, None]) & 1).double()
    d = -(de @ bit) + ((torch.triu(U, 1).T @ bit) * bit).sum(0)
    up = (0.5 * om * torch.exp(1j * ph))[:, None]
    with torch.no_grad():
        one = bit == 1

    def h(p):  # the flips' coefficients by the target bit
        g = p[idx]
        return d * p + (up * torch.where(one, g, 0.0)).sum(0) + (up.conj() * torch.where(one, 0.0, g)).sum(0)

    def step(p):  # the expansion again for the backward pass, a few terms at a time
        return torch.utils.checkpoint.checkpoint(h, p, use_reentrant=False)

    out = _expm(step, lo, hi, dt, psi)
    g = torch.autograd.grad(out, [*x, psi], s["w"].to(torch.complex128))
    return [out.detach(), *g]


def _exact_pulse(case, s):
    n, S = case["n"], case["sets"]
    D = 1 << n
    om, de = (torch.as_tensor(s[q], device=DEV).requires_grad_() for q in ("om", "de"))
    psi0 = torch.zeros(S, D, dtype=torch.complex128, device=DEV)
    psi0[:, 0] = 1.0
    psi0.requires_grad_()
    eu = _diagonal(np.zeros(n), s["U"], n)
    pop = _diagonal(-np.ones(n), np.zeros((n, n)), n)
    idx = _xor_index(n).reshape(-1)
    span = 0.5 * n * float(om.max()) + n * float(de.abs().max())
    lo, hi = float(eu.min()) - span, float(eu.max()) + span

    def step(p, o, e):
        def h(v):
            x = v[:, idx].view(S, n, D).sum(1)
            return (eu - e[:, None] * pop) * v + (0.5 * o)[:, None] * x
        return _expm(h, lo, hi, case["dt"], p)

    psi = psi0
    for j in range(case["segments"]):
        for _ in range(case["steps"]):
            psi = torch.utils.checkpoint.checkpoint(step, psi, om[:, j], de[:, j], use_reentrant=False)
    p2 = psi.real ** 2 + psi.imag ** 2
    occ = torch.stack([p2.view(S, 1 << i, 2, -1)[:, :, 1].sum((1, 2)) for i in range(n)], 1)
    loss = ((occ - torch.as_tensor(s["target"], device=DEV)) ** 2).mean(1)
    g = torch.autograd.grad(loss.sum(), [om, de, psi0])
    return [loss.detach(), *g]


def _exact_lindblad(case, s):
    n = case["n"]
    D = 1 << n
    ops = [L.to(DEV) for L in _lindblads()]
    h, lo, hi = _operator(s["om"], s["de"], s["ph"], s["U"], n)
    width = hi - lo
    noise = torch.as_tensor(_noise(), device=DEV)

    def on_rows(op, x, i):  # a 2 x 2 operator on qubit i of the row index
        return torch.einsum("ab,xby->xay", op, x.reshape(1 << i, 2, -1)).reshape(D, D)

    h_rows = _row_operator(s, n)

    def heff(x):
        a = h_rows(x)
        for i in range(n):
            a = a + on_rows(noise, x, i)
        return a

    def lind(rho):  # linear: the expansion's terms are not all Hermitian
        out = heff(rho) - heff(rho.conj().T.contiguous()).conj().T
        for i in range(n):
            for L in ops:
                t = on_rows(L, rho, i)
                out = out + 1j * on_rows(L.conj(), t.T.contiguous(), i).T
        return out

    return _expm(lind, -width, width, case["dt"], s["rho"].to(torch.complex128))


def _row_operator(s, n):
    """rho -> H rho (H on the row index)."""
    om, ph = s["om"].double().numpy(), s["ph"].double().numpy()
    d = _diagonal(s["de"].numpy(), s["U"].numpy(), n)
    up = 0.5 * om * np.exp(1j * ph)

    def h(rho):
        out = d[:, None] * rho
        for i in range(n):
            v, o = rho.reshape(1 << i, 2, -1), out.view(1 << i, 2, -1)
            o[:, 1] += complex(up[i]) * v[:, 0]
            o[:, 0] += complex(up[i].conjugate()) * v[:, 1]
        return out

    return h
