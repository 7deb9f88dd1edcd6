"""GPU: the expand-sort-compress CTA bins, whose radix sort takes the passes a
row's span of columns needs: spans around one, two and three passes of seven
bits, at offsets that are no multiple of them and at both ends of B.n, row sizes
around each kernel's limits, repeated columns and one column alone, against the
oracle: structure bit-exact, values within 1e-12 (FP64) or 1e-5 (FP32) of
sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu

SPANS = [1, 2, 127, 128, 129, 16383, 16384, 16385, 1 << 18, 1 << 20]
SIZES = [513, 1023, 1024, 1025, 2047, 2048, 2049, 3071, 3072]


def _operands(n, dtype):
    """A row of about every size over its own block of B rows, for every span."""
    rng = np.random.default_rng(n % 1009)
    a_rows, b_rows = [], []
    for span in (s for s in SPANS if s <= n):
        for size in SIZES:
            first = int(rng.choice([0, n - span, rng.integers(0, n - span + 1)]))
            at, left = len(b_rows), size
            ends = [[first], [first + span - 1]]
            while left > 0:
                k = min(left, int(rng.integers(1, 9)), span)
                c = ends.pop() if ends else np.unique(rng.integers(first, first + span, k))
                b_rows.append(np.asarray(c))
                left -= len(c)
            a_rows.append(np.arange(at, len(b_rows)))

    def csr(rows, cols):
        rpt = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
        col = np.concatenate(rows).astype(np.int32)
        return HostCSR(len(rows), cols, rpt, col, rng.uniform(-1, 1, col.size).astype(dtype))

    return csr(a_rows, len(b_rows)), csr(b_rows, n)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [129, 16385, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, 1 << 22])
def test_sort_span(handle, oracle_mod, n, dtype):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    A, B = _operands(n, dtype)
    handle.set_option(N.OPT_ONE_PASS, 1)
    handle.set_option(N.OPT_ESC, 1)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
        info = handle.info()
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)
        handle.set_option(N.OPT_ESC, 0)
    assert info["one_pass"] == 1 and info["esc_mask"] == 0b11111
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
    assert res["rpt_equal"] and res["col_equal"], res
    assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res
