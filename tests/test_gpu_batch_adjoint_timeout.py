"""A batched adjoint launch whose waits run out (emusv_batch_set_barrier_test on its workspace):
every register's status is EMUSV_TIMEOUT, whatever an earlier launch, or memory that was never
written, left in the bases' states; PulseGradientBatch raises TimeoutError, and the same workspace
then gives the gradients it gave before.  Registers run by gangs, and more tiles than warps (the
phase engine)."""

import numpy as np
import pytest
import torch

from emulators_b200 import _lib
from emulators_b200 import workloads as wl
from emulators_b200.gradients import PulseGradientBatch

pytestmark = pytest.mark.gpu


def _batch(n, sets, tile):
    rng = np.random.default_rng(n + sets)
    U = wl.interaction_matrix(wl.random_box(n, 60.0, 5.0, rng))
    om, de = rng.uniform(1.0, 6.0, (sets, 2)), rng.uniform(-8.0, 8.0, (sets, 2))
    target = (np.arange(n) % 2).astype(float)
    return PulseGradientBatch(U, 0.01, om, de, 2, target, tile_bits=tile)


@pytest.mark.parametrize("n,sets,tile", [(10, 3, 8), (12, 2, 9), (15, 12, 9)])
@pytest.mark.parametrize("first", [False, True])
def test_a_timeout_is_reported_and_recovered_from(n, sets, tile, first):
    b = _batch(n, sets, tile)
    L = _lib.load()
    if first:  # memory that reads as finished runs of one iteration
        b.ws_a.view(torch.int32).fill_(1)
        b.ws_f.view(torch.int32).fill_(1)
        s = torch.cuda.current_stream().cuda_stream
        a = (b.nsets, b.nq.ctypes.data, b.ns.ctypes.data, b.dts.ctypes.data, b.code, b.om.ctypes.data,
             b.de.ctypes.data, b.ph.ctypes.data, b.Us.ctypes.data)
        _lib.check(L.emusv_batch_prepare(*a, b.states.data_ptr(), b.tol, b.tol, b.maxdim, b.T, b.capacity,
                                         b.ws_f.data_ptr(), b.ws_f.numel(), s), "prepare")
        _lib.check(L.emusv_batch_adjoint_prepare(*a, b.tol, b.maxdim, b.T, b.capacity, b.ws_a.data_ptr(),
                                                 b.ws_a.numel(), s), "prepare")
    else:
        want = b.loss_and_grad()
    _lib.check(L.emusv_batch_set_barrier_test(b.ws_a.data_ptr(), 2_000_000, 1), "switch")
    with pytest.raises(TimeoutError):
        b.loss_and_grad()
    assert (b.status == _lib.TIMEOUT).all()
    _lib.check(L.emusv_batch_set_barrier_test(b.ws_a.data_ptr(), 0, 0), "switch")
    got = b.loss_and_grad()
    if first:
        want = _batch(n, sets, tile).loss_and_grad()
    for x, y in zip(got, want):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-9)
