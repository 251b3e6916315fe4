"""The Arnoldi step (without a noise term, so that the Lanczos oracle knows its result) at the sizes
where the Gram-Schmidt passes change: one chunk of amplitudes with the basis spread over blocks, a
block or two per SM, and a basis beyond the L2, whose update pass runs backwards; both precisions."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, krylov
from emulators_b200 import workloads as wl
from emulators_b200.krylov import fused_arnoldi_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dt", [(2, 0.02), (9, 0.03), (12, 0.02), (17, 0.01), (19, 0.01), (20, 0.01), (21, 0.006)])
def test_arnoldi_step_matches_oracle(oracle, n, dt):
    rng = np.random.default_rng(n)
    om, de, ph = rng.uniform(1.0, 6.0, n), rng.uniform(-8.0, 8.0, n), rng.uniform(0.0, 6.0, n)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    ref, _, res = oracle.evolve_step(dt, om, de, ph, U, psi, 1e-10)
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in (om, de, ph, U)), "cuda")
    krylov.release_workspaces()
    # both within the exponential's tolerance; complex64: about 30 vectors rounded at 2^-24, two
    # operations each
    for dtype, bar in ((torch.complex128, 2e-10), (torch.complex64, 5e-6)):
        out, info, st = fused_arnoldi_step(HamiltonianExpOperator(H, dt), torch.as_tensor(psi).to("cuda", dtype),
                                           1e-10, 1e-10, 100)
        assert st == 0 and np.linalg.norm(out.cpu().numpy() - ref) <= bar
        if dtype == torch.complex128:
            assert info.iterations == res.iteration_count
    krylov.release_workspaces()
