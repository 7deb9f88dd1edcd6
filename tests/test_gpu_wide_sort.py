"""GPU: expand-sort-compress and ranged-bitmap fills of a wide B (2^20 < B.n <=
2^22), around the widths where a key's column bits run out (2^20, 2^22) and the
row sizes where the kernels change, with columns at both ends of B.n, against
the oracle: structure bit-exact, values within 1e-12 (FP64) or 1e-5 (FP32) of
sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu

SIZES = [1, 11, 12, 13, 47, 49, 190, 193, 511, 513, 767, 769, 1023, 1025, 2047, 2049, 3071, 3073, 12287, 12289,
         30000]


def _operands(n, dtype, seed):
    """Rows of about SIZES products over B rows of 1 to 20 entries; some B rows
    share columns, some hold the first and the last columns of every 2^18."""
    rng = np.random.default_rng(seed)
    edges = np.unique(np.concatenate([np.arange(0, n, 1 << 18), np.arange(0, n, 1 << 18) - 1,
                                      [0, n - 1]]))
    edges = edges[(edges >= 0) & (edges < n)]
    b_rows = []
    for i in range(4000):
        k = int(rng.integers(1, 21))
        c = rng.choice(edges, min(k, edges.size), replace=False) if i % 50 == 0 else \
            rng.integers(0, n if i % 3 else 3000, k)
        b_rows.append(np.unique(c))
    lens = np.array([r.size for r in b_rows])
    a_rows = []
    for size in SIZES * 6:
        order = rng.permutation(4000)
        take = int(np.searchsorted(np.cumsum(lens[order]), size))
        a_rows.append(np.sort(order[:max(take, 1)]))
    a_rows += [np.sort(rng.choice(4000, int(rng.integers(0, 5)), replace=False))
               for _ in range(20000)]

    def csr(rows, cols):
        rpt = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
        col = np.concatenate(rows).astype(np.int32)
        return HostCSR(len(rows), cols, rpt, col, rng.uniform(-1, 1, col.size).astype(dtype))

    return csr(a_rows, 4000), csr(b_rows, n)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("esc", [0, 1])
@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1, (1 << 21) + 7, 1 << 22, (1 << 22) + 1])
def test_wide_sort(handle, oracle_mod, n, esc, dtype):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    A, B = _operands(n, dtype, n % 1000 + esc)
    handle.set_option(N.OPT_ONE_PASS, 1)
    handle.set_option(N.OPT_ESC, esc)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
        info = handle.info()
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)
        handle.set_option(N.OPT_ESC, 0)
    assert info["one_pass"] == 1
    if esc == 1:
        assert info["esc_mask"] == (0b11111 if n <= 1 << 22 else 0)
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
    assert res["rpt_equal"] and res["col_equal"], res
    assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res
