"""A step of a batch that reaches max_krylov_dim is reported (EMUSV_NOT_CONVERGED, the reference's
RecursionError) whichever step it is: here the first of three, the later ones converging in a few
iterations; lock-step rounds, gangs and (more tiles than warps) the phase engine."""

import numpy as np
import pytest

from emulators_b200 import workloads as wl
from emulators_b200.batch import BatchEvolution

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("sizes", [[10, 12, 11], [16] * 12])
def test_an_early_step_that_does_not_converge(sizes, engine):
    rng = np.random.default_rng(len(sizes))
    regs = []
    for i, n in enumerate(sizes):
        U = wl.interaction_matrix(wl.random_box(n, 300.0, 5.0, rng))
        om = np.full((3, n), 0.05)
        if i == 1:
            om[0] = 60.0
        regs.append(wl.Workload(f"r{n}", None, U, 0.01, om, np.zeros((3, n)), np.zeros((3, n))))
    b = BatchEvolution(regs, precision="c128", max_krylov_dim=10)
    b.prepare(9, 11)
    b.set_engine(engine)
    b.launch(1)
    status, iters = b.results(raise_on_error=False)
    assert iters[1, 0] == 10 and iters[1, 2] < 10
    assert status[1] == 1 and b.last_code == 1
    assert (np.delete(status, 1) == 0).all()
    with pytest.raises(RecursionError):
        b.run(tune=False, tile_bits=9, engine=engine)
