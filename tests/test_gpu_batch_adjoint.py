"""The batched adjoint step (emusv_batch_adjoint_launch) on registers of uneven size against the
one-register adjoint, at the sizes where its contraction kernels split their work: one block of
amplitudes and less (8-10 qubits), the groups of high bits (11, 14, 15) and several blocks that
share a tile's outputs; phases, and a register whose incoming gradient is zero."""

import numpy as np
import pytest
import torch

from emulators_b200 import _lib
from emulators_b200 import workloads as wl
from emulators_b200.adjoint import step_adjoint

pytestmark = pytest.mark.gpu
BMAXQ = 20
TOL = 1e-10


@pytest.mark.parametrize("dtype,tile", [(torch.complex128, 8), (torch.complex128, 9), (torch.complex64, 8),
                                        (torch.complex64, 9), (torch.complex64, 10)])
@pytest.mark.parametrize("sizes", [[10], [8, 9, 11, 10, 14, 8], [15, 10, 13], [12] * 40, [18, 10]])
def test_batched_adjoint_matches_the_single_one(dtype, tile, sizes):
    sizes = [max(n, tile) for n in sizes]
    rng = np.random.default_rng(31 * len(sizes) + tile)
    S, dt = len(sizes), 0.01
    L = _lib.load()
    om, de, ph, Us, st, gr = [], [], [], [], [], []
    for i, n in enumerate(sizes):
        pos = wl.random_box(n, 40.0, 5.0, rng)
        Us.append(wl.interaction_matrix(pos))
        om.append(rng.uniform(1.0, 6.0, n))
        de.append(rng.uniform(-10.0, 10.0, n))
        ph.append(rng.uniform(0.0, 6.0, n) * (i % 2))
        v = rng.normal(size=(2, 1 << n)) + 1j * rng.normal(size=(2, 1 << n))
        st.append(torch.tensor(v[0] / np.linalg.norm(v[0]), device="cuda").to(dtype))
        gr.append(torch.tensor(v[1] / np.linalg.norm(v[1]), device="cuda").to(dtype))
    zero = 1 if S > 1 else None
    if zero is not None:
        gr[zero].zero_()
    nq, ns = np.asarray(sizes, dtype=np.int32), np.ones(S, dtype=np.int32)
    dts = np.full(S, dt)
    code, cap = _lib.dtype_code(dtype), 40
    h = [np.ascontiguousarray(np.concatenate([x.reshape(-1) for x in a])) for a in (om, de, ph, Us)]
    nb = L.emusv_batch_adjoint_workspace_bytes(S, nq.ctypes.data, ns.ctypes.data, code, tile, cap)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    psi, gin = torch.cat(st), torch.cat(gr)
    gout = torch.full_like(gin, 7.0)
    grads = torch.full((S, 3, BMAXQ), 7.0, dtype=torch.float64, device="cuda")
    status = torch.full((S,), -1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    _lib.check(L.emusv_batch_adjoint_prepare(S, nq.ctypes.data, ns.ctypes.data, dts.ctypes.data, code,
                                             *(a.ctypes.data for a in h), TOL, 100, tile, cap,
                                             ws.data_ptr(), nb, s), "prepare")
    for _ in range(2):  # the second launch starts from the first one's hints and partials
        _lib.check(L.emusv_batch_adjoint_launch(code, tile, 1, 0, psi.data_ptr(), gin.data_ptr(),
                                                gout.data_ptr(), grads.data_ptr(), status.data_ptr(),
                                                ws.data_ptr(), s), "launch")
    assert (status == 0).all()
    got = [grads[i, :, :n].cpu().numpy() for i, n in enumerate(sizes)]
    outs = torch.split(gout, [1 << n for n in sizes])
    for i, n in enumerate(sizes):
        if i == zero:
            assert not got[i].any() and not outs[i].any()
            continue
        t = [torch.tensor(a[i]) for a in (om, de, ph, Us)]
        ref = step_adjoint(dt, *t, st[i], gr[i], TOL, 100, (True, True, True, False, True))
        # the bar of the one-register adjoint: max(10 tolerances, 1e-11) of scale >= 1 in
        # complex128, 1e-5 of it for vectors stored in complex64
        bar = 10 * TOL if dtype == torch.complex128 else 1e-5
        for a, b in zip((*got[i], outs[i].cpu().numpy()), (ref[0], ref[1], ref[2], ref[4])):
            b = b.detach().cpu().numpy()
            assert np.abs(a - b).max() <= bar * max(1.0, np.abs(b).max()), (i, n)
