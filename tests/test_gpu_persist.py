"""Time steps that run in one launch (registers up to 20 qubits), at the sizes where their
shape changes: fewer amplitudes than threads, one CTA, clusters of 8 and 16 CTAs, the whole
GPU, and 21 qubits, the first register beyond it."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, krylov
from emulators_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _case(n, phase, seed):
    rng = np.random.default_rng(seed)
    pos = wl.random_box(n, 40.0, 5.0, rng)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi *= np.exp(-rng.uniform(0.0, 8.0, size=1 << n))  # uneven amplitudes, as in a blockaded state
    ph = rng.uniform(0.0, 2.0 * np.pi, n) if phase else np.zeros(n)
    return np.full(n, 4.0), rng.uniform(-8.0, 8.0, n), ph, wl.interaction_matrix(pos), psi / np.linalg.norm(psi)


def _step(case, dtype, dt, maxdim=100):
    om, de, ph, U, psi = case
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in (om, de, ph, U)), "cuda")
    v = torch.as_tensor(psi, device="cuda").to(dtype)
    out, info, st = krylov.fused_step(HamiltonianExpOperator(H, dt), v, 1e-10, 1e-10, maxdim)
    return out.cpu().numpy(), info, st


@pytest.mark.parametrize("phase", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 21])
def test_step_matches_oracle(oracle, n, phase):
    case = _case(n, phase, 7 * n + phase)
    om, de, ph, U, psi = case
    dt = 0.004
    ref, _, res = oracle.evolve_step(dt, om, de, ph, U, psi, 1e-10)
    out, info, st = _step(case, torch.complex128, dt)
    assert st == 0 and info.iterations == res.iteration_count
    assert np.linalg.norm(out - ref) <= 2e-10  # both within the tolerance of the exponential
    assert abs(info.output_norm - np.linalg.norm(out)) <= 1e-12
    # complex64: about 25 vectors rounded at 2^-24, two operations each
    out64, _, st = _step(case, torch.complex64, dt)
    assert st == 0 and np.linalg.norm(out64 - ref) <= 4e-6


@pytest.mark.parametrize("n", [6, 11, 13, 16])
def test_basis_grows_beyond_its_first_capacity(oracle, n):
    case = _case(n, True, n)
    om, de, ph, U, psi = case
    krylov.release_workspaces()
    c = krylov._cache(torch.device("cuda", 0), n, 0)  # a first workspace of 8 vectors
    c.capacity, c.buf = 8, torch.zeros(1, dtype=torch.uint8, device="cuda")
    ref, _, res = oracle.evolve_step(0.05, om, de, ph, U, psi, 1e-10)
    assert res.iteration_count > 8
    out, info, st = _step(case, torch.complex128, 0.05)
    assert st == 0 and info.iterations == res.iteration_count
    assert np.linalg.norm(out - ref) <= 2e-10
    _, info, st = _step(case, torch.complex128, 0.05, maxdim=5)
    assert st == 1 and info.iterations == 5 and not info.converged


@pytest.mark.parametrize("n", [4, 11, 13, 17])
def test_states_that_end_a_run_early(n):
    om, de, ph, U, psi = _case(n, False, n)
    # an eigenvector of a diagonal Hamiltonian: happy breakdown in the first iteration
    e0 = np.zeros_like(psi)
    e0[5 % len(e0)] = 1.0
    out, info, st = _step((0 * om, de, ph, U, e0), torch.complex128, 0.01)
    assert st == 0 and info.happy_breakdown and info.iterations == 1
    assert abs(abs(out[5 % len(e0)]) - 1.0) <= 1e-14
    # zero and non-finite states
    for bad in (np.zeros_like(psi), np.where(np.arange(len(psi)) == 1, np.nan, psi)):
        with pytest.raises(FloatingPointError):
            _step((om, de, ph, U, bad), torch.complex128, 0.01)
    # and the next step is unharmed
    a, _, _ = _step((om, de, ph, U, psi), torch.complex128, 0.004)
    assert abs(np.linalg.norm(a) - 1.0) <= 1e-10
