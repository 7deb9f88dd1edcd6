"""GPU: the compression sample's sums, by the kernels they choose.  Rows whose
first B rows repeat their columns and whose next B row is long: the sample's
table cannot take that row, and its products must not count against the others.
Every row of A is sampled (2,048 rows), so the sampled ratio is exact: rows of 51
short B rows (15 of 30 columns) and rows of 16 short ones and one of `long`."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu

M, PER, N_LONG = 2048, 60, 40


def _operands(long, share, rng):
    n = 40_000
    b_rows = [np.sort(rng.choice(30, 15, replace=False)) for _ in range(PER)]
    b_rows += [30 + np.sort(rng.choice(2 * long, long, replace=False)) for _ in range(N_LONG)]
    is_long = np.zeros(M, bool)
    is_long[rng.choice(M, int(share * M), replace=False)] = True
    a_rows = [np.concatenate([np.sort(rng.choice(PER, 16, replace=False)),
                              [PER + int(rng.integers(N_LONG))]]) if x
              else np.sort(rng.choice(PER, 55, replace=False)) for x in is_long]

    def csr(rows, cols):
        rpt = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
        col = np.concatenate(rows).astype(np.int32)
        return HostCSR(len(rows), cols, rpt, col, rng.uniform(-1, 1, col.size))
    return csr(a_rows, PER + N_LONG), csr(b_rows, n), is_long


# a short row's 768 first products: 754 counted, 30 columns; a long row's: 240 + long
# counted, 30 + long columns.  The window bins start at a ratio of 1.5.
@pytest.mark.parametrize("long,share,windows", [(1100, 0.655, True), (2500, 0.34, True),
                                                (1100, 1.0, False), (2500, 1.0, False),
                                                (1100, 0.0, True), (520, 1.0, None)])
def test_long_b_row_at_the_cut(handle, oracle_mod, long, share, windows):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    A, B, is_long = _operands(long, share, np.random.default_rng(long))
    assert A.nnz > 1 << 15
    ratio = ((754 * (~is_long).sum() + (240 + long) * is_long.sum()) /
             (30 * (~is_long).sum() + (30 + long) * is_long.sum()))
    if windows is not None:
        assert (ratio >= 1.5) == windows  # the case is what it says
    handle.set_option(N.OPT_ONE_PASS, 1)
    handle.set_option(N.OPT_PROFILE, 1)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
        names = [k["name"] for k in handle.profile()]
    finally:
        handle.set_option(N.OPT_PROFILE, 0)
        handle.set_option(N.OPT_ONE_PASS, 0)
    if windows is not None:
        assert any(x.startswith("win_fill") for x in names) == windows, names
    R = oracle_mod.spgemm(A, B, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A, B, R))
    assert res["rpt_equal"] and res["col_equal"] and res.get("max_cond", 0.0) <= 1e-12, res
