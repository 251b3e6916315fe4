"""A recomputation of a checkpoint segment whose waits run out (the switch on the forward workspace,
set after the forward pass): the gradients of its states are not handed out, TimeoutError is raised,
and the next call gives the gradients it gave before."""

import numpy as np
import pytest

from emulators_b200 import _lib
from emulators_b200 import workloads as wl
from emulators_b200.gradients import PulseGradientBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [0, 1])
def test_a_recomputation_that_times_out(engine):
    n, sets = 10, 3
    rng = np.random.default_rng(4)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    om, de = rng.uniform(1.0, 6.0, (sets, 2)), rng.uniform(-8.0, 8.0, (sets, 2))
    b = PulseGradientBatch(U, 0.01, om, de, 3, (np.arange(n) % 2).astype(float), checkpoint_every=3, engine=engine)
    want = b.loss_and_grad()
    L = _lib.load()
    b.forward()
    occ = b.occupations()
    _lib.check(L.emusv_batch_set_barrier_test(b.ws_f.data_ptr(), 2_000_000, 1), "switch")
    with pytest.raises(TimeoutError):
        b.backward(occ)
    _lib.check(L.emusv_batch_set_barrier_test(b.ws_f.data_ptr(), 0, 0), "switch")
    for x, y in zip(b.loss_and_grad(), want):
        np.testing.assert_array_equal(x, y)
