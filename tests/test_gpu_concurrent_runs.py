"""Time steps from several threads, each on its own stream: one-launch runs of one CTA, of a cluster
and of the whole GPU side by side give the bits they give alone."""

import threading

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, krylov
from emulators_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _chain(n, steps):
    rng = np.random.default_rng(n)
    U = torch.as_tensor(wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng)))
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    for _ in range(steps):
        p = [torch.as_tensor(rng.uniform(lo, hi, n)) for lo, hi in ((1.0, 6.0), (-8.0, 8.0), (0.0, 6.0))]
        H = RydbergHamiltonian(*p, U, "cuda")
        psi, _, st = krylov.fused_step(HamiltonianExpOperator(H, 0.005), psi, 1e-10, 1e-10, 100)
        assert st == 0
    return psi


@pytest.mark.parametrize("sizes", [[16, 17, 18, 19], [10, 13, 15, 16, 20]])
def test_threads_on_their_own_streams(sizes):
    steps = 40
    krylov.release_workspaces()
    want = {n: _chain(n, steps) for n in sizes}
    krylov.release_workspaces()  # the energy shift starts anew
    torch.cuda.synchronize()
    got, errors = {}, []

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got[n] = _chain(n, steps)
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # reported by the main thread
            errors.append((n, e))

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for n in sizes:
        assert torch.equal(got[n], want[n]), n
