"""GPU: a product of a range of A's rows (A.rpt inside the matrix's, A.col and
A.val whole: what a batch's group is) runs the kernels that the same rows as a
matrix of their own do, and gives the same C."""
import numpy as np
import pytest

from test_gpu_window import _repeating

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [1, 2])
def test_same_kernels(handle, passes):
    import torch

    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    A, B = _repeating(120_000, 15, 190, 50_000, np.float64, 1)
    dA, dB = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
    r0, r1 = 60_000, 66_000
    e0, e1 = int(A.rpt[r0]), int(A.rpt[r1])
    assert e1 - e0 > 1 << 15 and A.nnz > 15 * (e1 - e0)
    view = DeviceCSR(r1 - r0, A.n, dA.rpt[r0:r1 + 1], dA.col, dA.val)
    alone = DeviceCSR(r1 - r0, A.n, dA.rpt[r0:r1 + 1] - e0, dA.col[e0:e1].clone(),
                      dA.val[e0:e1].clone())
    handle.set_option(N.OPT_ONE_PASS, passes)
    handle.set_option(N.OPT_PROFILE, 1)
    try:
        out = []
        for x in (alone, view):
            C = proposal(x, dB, handle)
            out.append((C, sorted((k["name"], k["rows"]) for k in handle.profile())))
    finally:
        handle.set_option(N.OPT_PROFILE, 0)
        handle.set_option(N.OPT_ONE_PASS, 0)
    (Ca, names_a), (Cv, names_v) = out
    assert any(n.startswith("win_fill") for n, _ in names_a), names_a
    assert names_v == names_a
    assert torch.equal(Ca.rpt, Cv.rpt) and torch.equal(Ca.col, Cv.col)
    assert torch.equal(Ca.val, Cv.val)  # the window bins add in one order
