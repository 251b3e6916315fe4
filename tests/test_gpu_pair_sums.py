"""Occupation, correlation, single-qubit density and sampling kernels at the register sizes
where their index split changes (fewer amplitudes than threads, one chunk, several chunks
without loop bits, every number of loop bits), against plain float64 sums."""

import numpy as np
import pytest
import torch

from emulators_b200.algebra import qubit_densities
from emulators_b200.observables import correlation, occupation
from emulators_b200.state_vector import sample_indices

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 10, 16, 17, 18, 19, 20, 21, 22, 23, 24]


def _state(n, dtype):
    g = torch.Generator(device="cuda").manual_seed(100 + n)
    v = torch.view_as_complex(torch.randn(1 << n, 2, dtype=torch.float64, device="cuda", generator=g))
    return (v / torch.linalg.vector_norm(v)).to(dtype)


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("n", SIZES)
def test_occupation_and_correlation(n, dtype):
    psi = _state(n, dtype)
    p = psi.to(torch.complex128).abs() ** 2
    occ, cor = occupation(psi).cpu(), correlation(psi).cpu()
    # sums of non-negative FP64 terms adding up to at most 1: both sides within 2^10 roundings
    tol = 1024 * np.finfo(np.float64).eps
    for i in range(n):
        pi = p.view(1 << i, 2, -1)[:, 1]
        assert abs(float(pi.sum()) - float(occ[i])) <= tol
        assert abs(float(pi.sum()) - float(cor[i, i])) <= tol
        for j in range(i + 1, n):
            ref = float(p.view(1 << i, 2, 1 << (j - i - 1), 2, -1)[:, 1, :, 1].sum())
            assert abs(ref - float(cor[i, j])) <= tol
            assert cor[i, j] == cor[j, i]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 11, 12, 13, 18])
def test_qubit_densities(n, dtype):
    psi = _state(n, dtype)
    rho = qubit_densities(psi).cpu()
    v = psi.to(torch.complex128)
    tol = 1024 * np.finfo(np.float64).eps
    for i in range(n):
        m = v.view(1 << i, 2, -1).transpose(0, 1).reshape(2, -1)
        assert (rho[i] - (m @ m.conj().T).cpu()).abs().max() <= tol


@pytest.mark.parametrize("n", [1, 4, 5, 8, 11, 12, 13, 17])
def test_sample_hits_the_index_of_every_interval(n):
    psi = _state(n, torch.complex128)
    p = (psi.abs() ** 2).cpu().numpy()
    cdf = np.cumsum(p)
    at = np.unique(np.linspace(0, (1 << n) - 1, 300).astype(np.int64))
    u = (cdf[at] - 0.5 * p[at]) / cdf[-1]  # the middle of each index's interval
    wide = p[at] > 1e-12  # rounding of the running sums stays far inside these intervals
    got = sample_indices(psi, torch.as_tensor(u)).cpu().numpy()
    assert (got[wide] == at[wide]).all() and wide.any()
