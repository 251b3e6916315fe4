"""The phase engine's bounded waits made to run out on a batch that it, and not the gangs, runs
(more tiles than warps): register 0's first phase is never published, every warp's starvation limit
runs out, the launch reports EMUSV_TIMEOUT, and the same workspace then gives the lock-step rounds'
bits."""

import numpy as np
import pytest
import torch

from emulators_b200 import workloads as wl
from emulators_b200.batch import BatchEvolution

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tile", [("c128", 9), ("c64", 8)])
def test_starvation_limit_runs_out_then_recovers(dtype, tile):
    rng = np.random.default_rng(tile)
    regs = []
    # 12 registers of 16 qubits in tiles of 2^9 amplitudes: 1536 tiles on at most 8 warps an SM (148
    # SMs); complex64 in tiles of 2^8, 3072 tiles on at most 16 warps an SM
    for n in [16] * 12:
        pos = wl.random_box(n, 60.0, 5.0, rng)
        om, de = rng.uniform(0.0, 6.0, (2, 1)), rng.uniform(-15.0, 15.0, (2, 1))
        regs.append(wl.Workload(f"r{n}", pos, wl.interaction_matrix(pos), 0.01, om * np.ones((1, n)),
                                de * np.ones((1, n)), np.zeros((2, n))))
    b = BatchEvolution(regs, precision=dtype)
    b.prepare(tile, 60)
    b.set_engine(1)
    b.set_barrier_test(wait_cycles=2_000_000, skip_first_arrival=True)
    b.launch(1)
    with pytest.raises(TimeoutError):
        b.results()
    b.set_barrier_test(0, False)
    got = []
    for engine in (1, 0):
        b.reset()
        b.set_engine(engine)
        b.launch(1)
        status, _ = b.results()
        assert (status == 0).all()
        got.append(b.states.clone())
    assert torch.equal(got[0], got[1])
