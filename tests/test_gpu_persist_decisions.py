"""Decisions of the one-launch time steps that are given up because an earlier iteration ended the
run: at every size class (one CTA, clusters, the whole GPU) a step taken again and again, while
deciding warps leave their exponentials at any point, gives the same bits."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, krylov
from emulators_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dt", [(9, 0.01), (11, 0.06), (12, 0.01), (15, 0.02), (16, 0.01), (18, 0.004)])
def test_a_step_repeats_to_the_bit(n, dt):
    rng = np.random.default_rng(n)
    om, de, ph = rng.uniform(0.0, 6.0, n), rng.uniform(-10.0, 10.0, n), rng.uniform(0.0, 6.0, n)
    U = wl.interaction_matrix(wl.random_box(n, 40.0, 5.0, rng))
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in (om, de, ph, U)), "cuda")
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    op = HamiltonianExpOperator(H, dt)
    krylov.release_workspaces()
    krylov.fused_step(op, psi, 1e-10, 1e-10, 100)  # the energy shift of the later steps
    first, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    assert st == 0
    for _ in range(200):
        out, again, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
        assert st == 0 and again.iterations == info.iterations
        assert torch.equal(out, first)
