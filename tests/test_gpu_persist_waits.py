"""The bounded waits of the one-launch runs made to run out (emusv_krylov_set_wait_test: one CTA
withholds its sums, the waits are cut to about a millisecond): the step and the adjoint step report
EMUSV_TIMEOUT (TimeoutError), the device stays usable and the next step on the same workspace
matches the oracle.  One CTA, clusters of 8 and 16, and the grid."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, _lib, krylov
from emulators_b200 import workloads as wl
from emulators_b200.adjoint import parameter_gradients

pytestmark = pytest.mark.gpu


@pytest.fixture
def withheld():
    yield lambda on: _lib.load().emusv_krylov_set_wait_test(2_000_000 if on else 0, int(on))
    _lib.load().emusv_krylov_set_wait_test(0, 0)


def _case(n):
    rng = np.random.default_rng(n)
    om, de, ph = rng.uniform(1.0, 6.0, n), rng.uniform(-8.0, 8.0, n), rng.uniform(0.0, 6.0, n)
    U = wl.interaction_matrix(wl.random_box(n, 40.0, 5.0, rng))
    v = rng.normal(size=(2, 1 << n)) + 1j * rng.normal(size=(2, 1 << n))
    return (om, de, ph, U), v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("n", [5, 11, 12, 15, 16, 19])
def test_step_times_out_and_recovers(oracle, withheld, n):
    p, v = _case(n)
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in p), "cuda")
    op, psi = HamiltonianExpOperator(H, 0.004), torch.as_tensor(v[0], device="cuda")
    krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    withheld(True)
    for _ in range(2):
        with pytest.raises(TimeoutError):
            krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    withheld(False)
    out, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    ref, _, res = oracle.evolve_step(0.004, *p, v[0], 1e-10)
    assert st == 0 and info.iterations == res.iteration_count
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 2e-10


@pytest.mark.parametrize("n", [9, 13, 17])
def test_adjoint_step_times_out_and_recovers(withheld, n):
    p, v = _case(n)
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in p), "cuda")
    psi, g = (torch.as_tensor(x, device="cuda") for x in v)
    want = parameter_gradients(H, 0.004, psi, g, 1e-10, 100)
    withheld(True)
    with pytest.raises(TimeoutError):
        parameter_gradients(H, 0.004, psi, g, 1e-10, 100)
    withheld(False)
    for a, b in zip(parameter_gradients(H, 0.004, psi, g, 1e-10, 100), want):
        np.testing.assert_array_equal(a, b)
