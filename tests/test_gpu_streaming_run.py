"""Krylov runs by the streaming passes: registers of 21 qubits, which always take them, and smaller
ones made to (emusv_krylov_set_streaming), as on a GPU that does not hold the one-launch run's
clusters.  Result and stopping iteration, the host's iteration hint, a basis that outgrows its
workspace, non-finite states, and the adjoint step."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, _lib, krylov
from emulators_b200 import workloads as wl
from emulators_b200.adjoint import parameter_gradients

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def streaming():
    _lib.load().emusv_krylov_set_streaming(1)
    krylov.release_workspaces()
    yield
    _lib.load().emusv_krylov_set_streaming(0)
    krylov.use_iteration_hint = True
    krylov.release_workspaces()


def _case(n, seed=0):
    rng = np.random.default_rng(n + seed)
    om, de, ph = rng.uniform(1.0, 6.0, n), rng.uniform(-8.0, 8.0, n), rng.uniform(0.0, 6.0, n) * (n % 2)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    v = rng.normal(size=(2, 1 << n)) + 1j * rng.normal(size=(2, 1 << n))
    return (om, de, ph, U), v / np.linalg.norm(v, axis=1, keepdims=True)


def _ham(p):
    return RydbergHamiltonian(*(torch.as_tensor(a) for a in p), "cuda")


@pytest.mark.parametrize("n", [12, 13, 16, 20, 21])
def test_step_matches_oracle(oracle, n):
    p, v = _case(n)
    ref, _, res = oracle.evolve_step(0.004, *p, v[0], 1e-10)
    op, psi = HamiltonianExpOperator(_ham(p), 0.004), torch.as_tensor(v[0], device="cuda")
    out, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    assert st == 0 and info.iterations == res.iteration_count
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 2e-10  # both within the exponential's tolerance
    _lib.load().emusv_krylov_set_streaming(0)  # the run by itself: the same iteration
    one, again, _ = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    assert again.iterations == info.iterations and float(torch.linalg.vector_norm(one - out)) <= 2e-10


@pytest.mark.parametrize("n", [13, 21])
def test_iteration_hint_keeps_counts_and_bits(n):
    """The host's read at every iteration, from the last count on, and far too late."""
    runs = []
    for mode in ("every", "hint", "high"):
        krylov.use_iteration_hint = mode != "every"
        krylov.release_workspaces()
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[0] = 1.0
        counts = []
        for k in range(6):
            if mode == "high" and counts:
                krylov._cache(psi.device, n, 0).last_iters = counts[-1] + 12
            psi, info, st = krylov.fused_step(HamiltonianExpOperator(_ham(_case(n, k)[0]), 0.01), psi, 1e-10, 1e-10, 100)
            assert st == 0
            counts.append(info.iterations)
        runs.append((psi, counts))
    for psi, counts in runs[1:]:
        assert counts == runs[0][1] and torch.equal(psi, runs[0][0])


@pytest.mark.parametrize("n", [13, 21])
def test_basis_grows_beyond_its_first_capacity(oracle, n):
    p, v = _case(n)
    c = krylov._cache(torch.device("cuda", 0), n, 0)
    c.capacity, c.buf = 8, torch.zeros(1, dtype=torch.uint8, device="cuda")
    ref, _, res = oracle.evolve_step(0.02, *p, v[0], 1e-10)
    assert res.iteration_count > 8
    op, psi = HamiltonianExpOperator(_ham(p), 0.02), torch.as_tensor(v[0], device="cuda")
    out, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    assert st == 0 and info.iterations == res.iteration_count
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 2e-10
    _, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 5)
    assert st == 1 and info.iterations == 5 and not info.converged


@pytest.mark.parametrize("n,dtype", [(13, torch.complex128), (16, torch.complex64), (21, torch.complex128)])
def test_nonfinite_and_zero_states(n, dtype):
    p, v = _case(n)
    op, psi = HamiltonianExpOperator(_ham(p), 0.004), torch.as_tensor(v[0], device="cuda").to(dtype)
    want, _, _ = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    bad = psi.clone()
    bad[5] = float("nan")
    for s in (bad, torch.zeros_like(psi)):
        with pytest.raises(_lib.NonFiniteError):
            krylov.fused_step(op, s, 1e-10, 1e-10, 100)
    krylov.release_workspaces()
    assert torch.equal(krylov.fused_step(op, psi, 1e-10, 1e-10, 100)[0], want)


@pytest.mark.parametrize("n", [12, 17])
def test_adjoint_step_matches_the_one_launch_bases(n):
    p, v = _case(n)
    psi, g = (torch.as_tensor(x, device="cuda") for x in v)
    got = parameter_gradients(_ham(p), 0.004, psi, g, 1e-10, 100)
    _lib.load().emusv_krylov_set_streaming(0)
    for a, b in zip(got, parameter_gradients(_ham(p), 0.004, psi, g, 1e-10, 100)):
        assert np.abs(a - b).max() <= 10 * 1e-10 * max(1.0, np.abs(b).max())  # the adjoint's bar
