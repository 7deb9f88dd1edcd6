"""GPU: the column-window bins (rows that repeat their columns inside a narrow
window of B) against the oracle, over every lane count (B rows of 1 to 100
entries, past a team's width too), windows of one word to their widest, both
value types, one pass and two, plans included; and rows that do not fit: wider
than the sampled window, more columns than the sampled compression says, and
B rows that are not sorted.  Tolerances are the parity tests': structure
bit-exact, values within 1e-12 (FP64) or 1e-5 (FP32) of sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu


def _csr(rows, n, rng, dtype):
    rpt = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32) if len(rows) else np.zeros(0, np.int32)
    return HostCSR(len(rows), n, rpt, col, rng.uniform(-1, 1, col.size).astype(dtype))


def _repeating(m, b_len, width, n, dtype, seed, a_len=40):
    """C rows of up to `width` columns hit many times: the B rows of a group
    hold about b_len columns of one window of `width`, and a row of A takes
    a_len rows of a group."""
    rng = np.random.default_rng(seed)
    groups, per = 20, 60
    b_rows = []
    for g in range(groups):
        base = 0 if g == 0 else n - width if g == 1 else int(rng.integers(0, n - width + 1))
        for _ in range(per):
            k = int(np.clip(rng.integers(b_len // 2, b_len + b_len // 2 + 1), 1, width))
            b_rows.append(base + np.sort(rng.choice(width, k, replace=False)))
    a_rows = []
    for r in range(m):
        k = int(rng.integers(1, a_len + 1)) if r % 7 else 0
        g = int(rng.integers(0, groups))
        a_rows.append(g * per + np.sort(rng.choice(per, k, replace=False)))
    return _csr(a_rows, groups * per, rng, dtype), _csr(b_rows, n, rng, dtype)


def _check(handle, oracle_mod, A, B, dtype, planned=False):
    from gpuspgemm_b200.api import DeviceCSR, plan, proposal
    dA, dB = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
    if planned:
        pl = plan(dA, dB, handle=handle)
        pl.result.val.zero_()
        pl.execute()
        pl.check()
        C = pl.result.to_host()
        pl.close()
    else:
        C = proposal(dA, dB, handle).to_host()
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
    assert res["rpt_equal"] and res["col_equal"], res
    assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res


def _uses_windows(handle, run):
    from gpuspgemm_b200 import _native as N
    handle.set_option(N.OPT_PROFILE, 1)
    try:
        run()
        return any(k["name"].startswith("win_fill") for k in handle.profile())
    finally:
        handle.set_option(N.OPT_PROFILE, 0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("b_len,width", [(2, 8), (3, 12), (3, 32), (4, 40), (7, 30), (8, 48),
                                         (14, 48), (6, 150), (15, 190), (27, 190), (30, 380),
                                         (16, 384), (30, 700), (100, 760)])
@pytest.mark.parametrize("passes", [1, 2])
def test_window_bins(handle, oracle_mod, b_len, width, passes, dtype):
    from gpuspgemm_b200 import _native as N
    A, B = _repeating(6000, b_len, width, 50_000, dtype, 100 * b_len + width)
    assert A.nnz >= 1 << 16  # sampled
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        used = _uses_windows(handle, lambda: _check(handle, oracle_mod, A, B, dtype))
        # (in one pass the smallest rows expand, sort and compress; the sample
        # sees the first 768 products of a row, which repeat little of 700 columns)
        assert used or passes == 1 or width > 400
        if passes == 2:
            _check(handle, oracle_mod, A, B, dtype, planned=True)
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)


@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("stretch", [30, 85, 120])
def test_window_widths(handle, oracle_mod, stretch, passes):
    """Columns spread by `stretch`: windows of 700 stretch columns, up to the
    widest bitmap (65,536 columns less the spare) and past it."""
    from gpuspgemm_b200 import _native as N
    A, B = _repeating(4200, 30, 700, 5000, np.float64, stretch)
    B = HostCSR(B.m, 5000 * stretch, B.rpt, (B.col * stretch + stretch - 1).astype(np.int32), B.val)
    assert A.nnz >= 1 << 16
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        _check(handle, oracle_mod, A, B, np.float64)
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("kind", ["wider", "more", "unsorted"])
def test_rows_that_do_not_fit(handle, oracle_mod, kind, passes, dtype):
    """Most rows repeat a few columns of a narrow window; every 61st (the
    sample's rows are evenly spread) does not."""
    from gpuspgemm_b200 import _native as N
    rng = np.random.default_rng(9)
    n, per = 60_000, 60
    b_rows = [np.sort(rng.choice(30, 12, replace=False)) for _ in range(per)]
    for _ in range(4000):
        if kind == "wider":
            b_rows.append(np.sort(rng.choice(n, 12, replace=False)))
        elif kind == "more":
            b_rows.append(np.sort(rng.choice(400, 12, replace=False)))
        else:
            b_rows.append(rng.choice(30, 12, replace=False))
    a_rows = []
    for r in range(8191):
        if r % 61 == 60:
            a_rows.append(per + np.sort(rng.choice(4000, 58, replace=False)))
        else:
            a_rows.append(np.sort(rng.choice(per, int(rng.integers(17, 50)), replace=False)))
    A, B = _csr(a_rows, per + 4000, rng, dtype), _csr(b_rows, n, rng, dtype)
    assert A.nnz >= 1 << 16
    handle.set_option(N.OPT_ONE_PASS, passes)
    try:
        _check(handle, oracle_mod, A, B, dtype)
    finally:
        handle.set_option(N.OPT_ONE_PASS, 0)
