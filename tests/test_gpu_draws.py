"""Bitstring draws against the inverse CDF in FP64, for the numbers of draws and sizes at which a draw
takes its groups of amplitudes one or eight at a time: the same index either way."""

import numpy as np
import pytest
import torch

from emulators_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [1, 4, 6, 7, 9, 11, 12, 13])
def test_draws_match_the_cdf(n, dtype):
    rng = np.random.default_rng(n)
    psi = torch.as_tensor(rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)).to("cuda", dtype)
    p = np.abs(psi.cpu().numpy().astype(np.complex128)) ** 2
    cdf = np.cumsum(p)
    L, code = _lib.load(), _lib.dtype_code(dtype)
    nb = L.emusv_sample_scratch_bytes(n)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    few = None
    u_all = rng.uniform(size=70000)
    for shots in (1, 500, 70000):
        u = torch.as_tensor(u_all[:shots].copy(), device="cuda")
        got = torch.empty(shots, dtype=torch.int64, device="cuda")
        _lib.check(L.emusv_sample(n, code, psi.data_ptr(), shots, u.data_ptr(), got.data_ptr(), scratch.data_ptr(), nb,
                                  _lib.stream_of(psi)), "sample")
        got = got.cpu().numpy()
        t = u_all[:shots] * cdf[-1]
        want = np.minimum(np.searchsorted(cdf, t, side="right"), (1 << n) - 1)
        # the device adds in another order: an index may be the neighbour where the target lies within
        # the sums' rounding (2^13 additions of 2^-53) of the step between them
        off = np.flatnonzero(got != want)
        edge = np.abs(cdf[np.minimum(got[off], want[off])] - t[off])
        assert (np.abs(got[off] - want[off]) == 1).all() and (edge <= cdf[-1] * (1 << n) * 2.0**-53).all()
        if few is not None:
            np.testing.assert_array_equal(got[: len(few)], few)  # the same draws by either way
        few = got
