"""Registers run by gangs (every tile of the batch has a warp of its own) against the lock-step
rounds: the same tiles' arithmetic and the same order of sums, so the same bits, at sizes from
one tile to several CTAs a register, with uneven step counts, and one batch beyond the warps of
the GPU (the phase engine)."""

import numpy as np
import pytest
import torch

from emulators_b200 import workloads as wl
from emulators_b200.batch import BatchEvolution

pytestmark = pytest.mark.gpu


def _batch(sizes, steps, dtype, seed):
    rng = np.random.default_rng(seed)
    regs = []
    for n, k in zip(sizes, steps):
        pos = wl.random_box(n, 40.0, 5.0, rng)
        om, de = rng.uniform(0.0, 6.0, (k, 1)), rng.uniform(-15.0, 15.0, (k, 1))
        ph = rng.uniform(0.0, 6.0, (1, n)) * np.ones((k, 1)) * (seed % 2)
        regs.append(wl.Workload(f"r{n}", pos, wl.interaction_matrix(pos), 0.01, om * np.ones((1, n)),
                                de * np.ones((1, n)), ph))
    return BatchEvolution(regs, precision=dtype)


@pytest.mark.parametrize("dtype,tile", [("c128", 8), ("c128", 9), ("c64", 8), ("c64", 9), ("c64", 10)])
@pytest.mark.parametrize("sizes,steps", [
    ([10], [3]),
    ([10, 11, 13, 14, 10], [4, 2, 4, 1, 3]),  # registers that end before the launch does
    ([12] * 9, [3] * 9),                       # more than one deciding CTA
    ([15, 10], [2, 3]),
    ([16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 16, 17], [2] * 12),  # more tiles than warps
])
def test_gangs_give_the_bits_of_the_rounds(dtype, tile, sizes, steps):
    b = _batch(sizes, steps, dtype, len(sizes) + tile)
    got = []
    for engine in (0, 1):
        status, iters = b.run(tune=False, tile_bits=tile, blocks_per_sm=1, capacity=60, engine=engine)
        assert (status == 0).all()
        taken = [iters[i, :k].copy() for i, k in enumerate(steps)]
        got.append((b.states.clone(), taken))
    assert torch.equal(got[0][0], got[1][0])
    for x, y in zip(got[0][1], got[1][1]):
        np.testing.assert_array_equal(x, y)


def test_gangs_report_a_basis_that_is_too_small():
    b = _batch([10, 12], [3, 3], "c128", 3)
    b.reset()
    b.prepare(9, 4)
    b.set_engine(1)
    b.launch(1)
    status, _ = b.results(raise_on_error=False)
    assert (status == 4).all()  # EMUSV_WORKSPACE_TOO_SMALL, as the rounds report it
    status, _ = b.run(tune=False, tile_bits=9, blocks_per_sm=1, capacity=4, engine=1)  # grown and retried
    assert (status == 0).all()
