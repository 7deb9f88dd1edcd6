"""GPU: the bitmap bin over a narrow B, whose threads hold blocks of four words
up to 2^19 columns and of 32 words past them: widths around a word, around four
words a thread for all threads and around the line between the two, columns at
both ends of B.n, row sizes from one product up to many chunks of A entries, one
row a CTA and more rows than CTAs, against the oracle: structure bit-exact,
values within 1e-12 (FP64) or 1e-5 (FP32) of sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu


def _operands(n, rows, dtype):
    rng = np.random.default_rng(n % 997 + rows)
    edges = np.unique(np.concatenate([np.arange(0, n, max(n // 8, 32)) + d for d in (-1, 0, 31, 32)]
                                     + [[0, n - 1]]))
    edges = edges[(edges >= 0) & (edges < n)]
    inner = 20000
    b_rows = [rng.choice(edges, min(4, edges.size), replace=False) if i % 10 == 0 else
              rng.integers(0, n, int(rng.integers(0, 6))) for i in range(inner)]
    b_rows = [np.unique(c) for c in b_rows]
    sizes = [1, 7, 1023, 1025, 8191, 8193, 20000]
    a_rows = [np.sort(rng.choice(inner, sizes[(i + rows) % len(sizes)], replace=False))
              for i in range(rows)]

    def csr(parts, cols):
        rpt = np.concatenate([[0], np.cumsum([r.size for r in parts])]).astype(np.int32)
        col = np.concatenate(parts).astype(np.int32)
        return HostCSR(len(parts), cols, rpt, col, rng.uniform(-1, 1, col.size).astype(dtype))

    return csr(a_rows, inner), csr(b_rows, n)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("rows", [1, 150])
@pytest.mark.parametrize("n", [1, 33, 1000, 1 << 17, (1 << 17) + 1, 1 << 19, (1 << 19) + 1])
def test_narrow_bitmap(handle, oracle_mod, n, rows, passes, dtype):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    A, B = _operands(n, rows, dtype)
    assert len(handle.ladder(2, 8)) == 7
    handle.set_option(N.OPT_MIN_NUM_BIN, 5)
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
    finally:
        handle.set_option(N.OPT_MIN_NUM_BIN, -1)
        handle.set_option(N.OPT_ONE_PASS, 0)
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
    assert res["rpt_equal"] and res["col_equal"], res
    assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res
