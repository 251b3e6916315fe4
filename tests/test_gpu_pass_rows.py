"""H*psi where the strided passes change their row width (64, 128 or 256 bytes
by the number of bits above the first pass), real and complex coefficients, noise term."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(17, torch.complex128), (18, torch.complex128), (19, torch.complex128),
                                     (22, torch.complex128), (25, torch.complex128), (18, torch.complex64),
                                     (19, torch.complex64), (20, torch.complex64), (22, torch.complex64),
                                     (25, torch.complex64)])
@pytest.mark.parametrize("phase,noisy", [(False, False), (True, False), (True, True)])
def test_row_widths_vs_oracle(oracle, n, dtype, phase, noisy):
    from emulators_b200 import RydbergHamiltonian
    from emulators_b200 import workloads as wl

    rng = np.random.default_rng(100 + n)
    om, de = rng.uniform(0, 2 * np.pi, n), rng.uniform(-20, 20, n)
    ph = rng.normal(size=n) if phase else np.zeros(n)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    noise = np.array([[0.1 - 0.2j, 0.05j], [-0.05j, 0.3 - 0.4j]]) if noisy else None
    psi = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) / np.sqrt(2 << n)
    kw = {"noise": noise} if noisy else {}
    ref = oracle.Hamiltonian(om, de, ph, U, **kw).apply(psi)
    kw = {"noise": torch.as_tensor(noise)} if noisy else {}
    H = RydbergHamiltonian(*(torch.as_tensor(a) for a in (om, de, ph, U)), "cuda", **kw)
    out = (H * torch.as_tensor(psi).to("cuda", dtype)).cpu().numpy()
    # the bar of the other layouts: 1e-13 of the largest component (23 flips and ~250 pair terms
    # of rounding 1.1e-16 each, relative to the component's own scale)
    # complex64 vectors: 1e-6 of it, a few of their roundings
    tol = 1e-13 if dtype == torch.complex128 else 1e-6
    np.testing.assert_allclose(out, ref, atol=tol * np.abs(ref).max(), rtol=0)
