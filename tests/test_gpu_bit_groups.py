"""Energy moments and time steps of product states at the register sizes where the strided passes
in front of the recurrence split the bits above its tile in another way: one group, two groups with
rows of 256, 128 and 64 bytes (21 to 29 qubits) and of 32 bytes (30 qubits).  Without interactions
the moments and the evolved state of a product state are known from its single qubits."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, StateVector, krylov

pytestmark = pytest.mark.gpu
X, Y = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]])


def _register(n, phase):
    rng = np.random.default_rng(3 * n + phase)
    om, de = rng.uniform(1.0, 2 * np.pi, n), rng.uniform(-5.0, 5.0, n)
    ph = rng.uniform(0.0, 2 * np.pi, n) if phase else np.zeros(n)
    h = [om[q] / 2 * (np.cos(ph[q]) * X + np.sin(ph[q]) * Y) - de[q] * np.diag([0, 1]) for q in range(n)]
    f = rng.normal(size=(n, 2)) + 1j * rng.normal(size=(n, 2))
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in (om, de, ph, np.zeros((n, n)))), "cuda")
    return H, h, f / np.linalg.norm(f, axis=1, keepdims=True)


def _product(f, dtype):
    v = torch.ones(1, dtype=dtype, device="cuda")
    for q in f:
        v = torch.outer(v, torch.as_tensor(q).to("cuda", dtype)).reshape(-1)
    return v


@pytest.fixture(autouse=True)
def _memory():
    yield
    krylov.release_workspaces()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,phase", [(13, True), (20, False), (21, True), (27, False), (28, True), (29, False),
                                     (30, True), (30, False)])
def test_moments_of_a_product_state(n, phase, dtype):
    H, h, f = _register(n, phase)
    psi = StateVector(_product(f, dtype))
    one = np.array([np.vdot(f[q], h[q] @ f[q]).real for q in range(n)])
    two = np.array([np.vdot(h[q] @ f[q], h[q] @ f[q]).real for q in range(n)])
    energy, second = one.sum(), one.sum() ** 2 + (two - one**2).sum()
    # an amplitude is a product of n rounded factors and enters twice; H psi adds about n roundings;
    # absolute against the sum of the terms' sizes
    eps = np.finfo(np.float32 if dtype == torch.complex64 else np.float64).eps
    bar, scale = 4 * n * eps, np.sqrt(two).sum()
    assert abs(float(H.expect(psi)) - energy) <= bar * scale
    assert abs(float(H.second_moment(psi)) - second) <= 2 * bar * scale**2


@pytest.mark.parametrize("n,phase", [(21, False), (28, True), (29, True), (30, False), (30, True)])
def test_step_of_a_product_state(n, phase):
    H, h, f = _register(n, phase)
    dt, dtype = 0.001, torch.complex64
    out, info, st = krylov.fused_step(HamiltonianExpOperator(H, dt), _product(f, dtype), 1e-8, 1e-8, 10)
    assert st == 0
    ev = []
    for q in range(n):
        e, V = np.linalg.eigh(h[q])
        ev.append(V @ (np.exp(-1j * dt * e) * (V.conj().T @ f[q])))
    ref = _product(ev, dtype)
    # both states are products of n rounded factors, the step adds a few roundings an iteration
    bar = (4 * n + 8 * info.iterations) * np.finfo(np.float32).eps
    assert float(torch.linalg.vector_norm(ref.sub_(out))) <= bar
