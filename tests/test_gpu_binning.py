"""GPU: the binning passes at the edges of their ranges.

Row counts around a CTA's rows (256), a scan tile (1,024) and the largest count
that the one-launch passes take (2^22), with rows of every fill list's limit
and one past it, in one pass and in two: every row of A holds one entry, so C's
rows are scaled rows of B and the comparison is exact.  Then rows of A at the
limits of the NIP pass's three row classes, against the oracle."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 12, 13, 48, 49, 192, 193, 512, 513, 768, 769, 1024, 1025, 2048, 2049, 3072, 3073]


@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("m", [1, 255, 256, 257, 1024, 1025, 606208, 4194304, 4194305])
def test_binning_row_counts(handle, m, passes):
    import torch

    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    rng = np.random.default_rng(m)
    n = 5000
    b_len = np.array(LENGTHS)
    b_rpt = np.concatenate([[0], np.cumsum(b_len)]).astype(np.int32)
    b_col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in b_len])
    pick = np.ones(m, np.int64)  # row 1 of B (one entry), but for a few
    some = rng.choice(m, size=min(m, 400), replace=False)
    pick[some] = rng.integers(0, len(LENGTHS), some.size)
    B = DeviceCSR.from_host(HostCSR(b_len.size, n, b_rpt, b_col.astype(np.int32),
                                    rng.uniform(0.5, 1.0, b_col.size)))
    A = DeviceCSR.from_host(HostCSR(m, b_len.size, np.arange(m + 1, dtype=np.int32),
                                    pick.astype(np.int32), rng.uniform(0.5, 1.0, m)))
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        C = proposal(A, B, handle)
        assert handle.info()["one_pass"] == (passes == 1)
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)
    row_len = torch.from_numpy(b_len).cuda()[A.col.long()]
    rpt = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rpt[1:] = torch.cumsum(row_len, 0)
    rows = torch.arange(m, device="cuda").repeat_interleave(row_len)
    at = torch.arange(rows.numel(), device="cuda") - rpt[rows] + B.rpt[A.col[rows].long()].long()
    assert torch.equal(C.rpt.long(), rpt)
    assert torch.equal(C.col, B.col[at])
    assert torch.equal(C.val, A.val[rows] * B.val[at])


@pytest.mark.parametrize("passes", [1, 2])
def test_nip_row_classes(handle, oracle_mod, passes):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200 import generators as G
    from gpuspgemm_b200.api import DeviceCSR, proposal
    rng = np.random.default_rng(5)
    k = 5000
    lens = rng.permutation(np.concatenate([np.repeat([31, 32, 33, 127, 128, 129, 513], 5), [4096, 0],
                                           rng.integers(0, 6, 300)]))
    cols = np.concatenate([np.sort(rng.choice(k, x, replace=False)) for x in lens])
    rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    A = HostCSR(lens.size, k, rpt, cols.astype(np.int32), rng.uniform(0.1, 1.0, cols.size))
    B = G.uniform_rows(3000, 3, seed=6, m=k)
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
        info = handle.info()
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)
    nip = oracle_mod.nip(A, B, per_row=True)[1]
    assert info["nip"] == int(nip.sum()) and info["max_row_nip"] == int(nip.max())
    R = oracle_mod.spgemm(A, B, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A, B, R))
    assert res["rpt_equal"] and res["col_equal"] and res.get("max_cond", 0.0) <= 1e-12, res
