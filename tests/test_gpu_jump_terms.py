"""The jump term of the Lindbladian for jump operators with few and many entries (one to twelve off
the diagonal of K = sum L (x) conj(L)): the walk by entry and, for many entries or few qubits, the
walk by qubit; against the oracle."""

import numpy as np
import pytest
import torch

from emulators_b200 import workloads as wl
from emulators_b200.density_matrix import RydbergLindbladian

pytestmark = pytest.mark.gpu
A, B, C, D = 0.3 - 0.1j, 0.5j, 0.2, -0.4
OPS = {
    "dephasing": [[[A, 0], [0, D]]],
    "relaxation": [[[0, B], [0, 0]]],
    "both ways": [[[0, B], [0, 0]], [[0, 0], [C, 0]]],
    "flip": [[[0, B], [C, 0]]],
    "upper": [[[A, B], [0, D]]],
    "three entries": [[[0, B], [C, D]]],
    "full": [[[A, B], [C, D]], [[0, 0.1], [0.7, 0]]],
}


@pytest.mark.parametrize("ops", list(OPS))
@pytest.mark.parametrize("n", [1, 2, 6, 7, 8])
def test_lindbladian_matches_oracle(oracle, n, ops):
    rng = np.random.default_rng(n)
    om, de, ph = rng.uniform(0.0, 6.0, n), rng.uniform(-10.0, 10.0, n), rng.normal(size=n)
    U = wl.interaction_matrix(wl.chain(n, 6.0))
    a = rng.normal(size=(1 << n, 3)) + 1j * rng.normal(size=(1 << n, 3))
    rho = a @ a.conj().T
    rho /= np.trace(rho).real
    L = [np.asarray(x, dtype=np.complex128) for x in OPS[ops]]
    ref = oracle.lindbladian_apply(om, de, ph, U, L, rho)
    op = RydbergLindbladian(*(torch.as_tensor(x) for x in (om, de, ph)), [torch.as_tensor(x) for x in L],
                            torch.as_tensor(U), "cuda")
    for dtype, tol in ((torch.complex128, 1e-12), (torch.complex64, 2e-6)):  # the bars of the other sizes
        got = (op @ torch.as_tensor(rho).to("cuda", dtype)).cpu().numpy()
        np.testing.assert_allclose(got, ref, atol=tol * np.abs(ref).max(), rtol=0)
