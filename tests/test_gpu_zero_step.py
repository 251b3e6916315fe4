"""A time step of length zero: the state itself after one iteration (the operator's norm is below
any tolerance, krylov_exp.py:60-71) and zero parameter gradients, for the one-launch runs, the
streaming run, the adjoint and the batches."""

import numpy as np
import pytest
import torch

from emulators_b200 import HamiltonianExpOperator, RydbergHamiltonian, krylov
from emulators_b200 import workloads as wl
from emulators_b200.adjoint import step_adjoint
from emulators_b200.batch import BatchEvolution

pytestmark = pytest.mark.gpu


def _case(n):
    rng = np.random.default_rng(n)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    p = [torch.as_tensor(a) for a in (rng.uniform(1.0, 6.0, n), rng.uniform(-8.0, 8.0, n), np.zeros(n), U)]
    v = rng.normal(size=(2, 1 << n)) + 1j * rng.normal(size=(2, 1 << n))
    return p, (torch.as_tensor(x / np.linalg.norm(x), device="cuda") for x in v)


@pytest.mark.parametrize("n", [1, 4, 11, 13, 17, 21])
def test_step_and_adjoint(n):
    p, (psi, g) = _case(n)
    op = HamiltonianExpOperator(RydbergHamiltonian(*p, "cuda"), 0.0)
    out, info, st = krylov.fused_step(op, psi, 1e-10, 1e-10, 100)
    assert st == 0 and info.happy_breakdown and info.iterations == 1
    # the normalised vector times the norm: a few roundings
    assert float((out - psi).abs().max()) <= 1e-15
    if n <= 17:
        got = step_adjoint(0.0, *p, psi, g, 1e-10, 100, (True, True, True, True, True))
        assert not any(x.abs().max() for x in got[:4])
        assert float((got[4] - g).abs().max()) <= 1e-15


@pytest.mark.parametrize("engine", [0, 1])
def test_batch(engine):
    regs = []
    for n, dt in ((9, 0.0), (10, 0.01), (11, 0.0)):
        pos = wl.random_box(n, 60.0, 5.0, np.random.default_rng(n))
        regs.append(wl.Workload(f"r{n}", pos, wl.interaction_matrix(pos), dt, np.ones((2, n)), np.ones((2, n)),
                                np.zeros((2, n))))
    b = BatchEvolution(regs, precision="c128")
    b.run(tune=False, tile_bits=8, blocks_per_sm=1, capacity=40, engine=engine)
    assert torch.isfinite(torch.view_as_real(b.states)).all()
    for i in (0, 2):
        o = int(b.offsets[i])
        first = b.initial[o:o + int(b.sizes[i])]
        assert float((b.state(i) - first).abs().max()) <= 1e-15
