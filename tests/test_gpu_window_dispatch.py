"""GPU: which kernels rows that repeat their columns run on, and that the rows that
do not fit them (in the unsampled places) were given to them first: then only the
fail list's hash kernel can have filled them.  Against the oracle: structure
bit-exact, values within 1e-12 (FP64) or 1e-5 (FP32) of sum |a||b|."""
import numpy as np
import pytest

from test_gpu_window import _csr

pytestmark = pytest.mark.gpu

SAMPLES = 2048


def _unsampled(m, step):
    """Every step-th row, but for the sampled ones and their neighbours."""
    sampled = (np.arange(SAMPLES, dtype=np.int64) * m) // SAMPLES
    rows = np.arange(step - 1, m, step)
    return rows[~np.isin(rows, np.concatenate([sampled - 1, sampled, sampled + 1]))]


def _check(handle, oracle_mod, A, B, dtype, passes, planned=False):
    """The kernels of one product, name -> rows."""
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, plan, proposal
    dA, dB = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
    handle.set_option(N.OPT_ONE_PASS, passes)
    handle.set_option(N.OPT_PROFILE, 1)
    try:
        C = proposal(dA, dB, handle).to_host()
        names = {}
        for k in handle.profile():
            names[k["name"]] = names.get(k["name"], 0) + k["rows"]
        results = [C]
        if planned:
            pl = plan(dA, dB, handle=handle)
            pl.result.val.zero_()
            pl.execute()
            pl.check()
            results.append(pl.result.to_host())
            pl.close()
    finally:
        handle.set_option(N.OPT_PROFILE, 0)
        handle.set_option(N.OPT_ONE_PASS, 0)
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    for C in results:
        res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
        assert res["rpt_equal"] and res["col_equal"], res
        assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res
    return names


def _rows(names, prefix):
    return sum(r for k, r in names.items() if k.startswith(prefix))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("kind", ["fits", "wider", "more", "unsorted"])
def test_rows_off_the_window(handle, oracle_mod, kind, passes, dtype):
    rng = np.random.default_rng(17)
    m, n, per = 16_381, 60_000, 60
    b_rows = [np.sort(rng.choice(30, 12, replace=False)) for _ in range(per)]
    for _ in range(4000):
        b_rows.append(np.sort(rng.choice(n, 12, replace=False)) if kind == "wider"
                      else np.sort(rng.choice(400, 12, replace=False)) if kind == "more"
                      else rng.choice(30, 12, replace=False) if kind == "unsorted"
                      else np.sort(rng.choice(30, 12, replace=False)))
    # 204 to 588 products a row: one fill bin in one pass
    a_rows = [np.sort(rng.choice(per, int(rng.integers(17, 50)), replace=False)) for _ in range(m)]
    off = _unsampled(m, 61)
    for r in off:
        a_rows[r] = per + np.sort(rng.choice(4000, 49, replace=False))
    assert off.size > 50
    A, B = _csr(a_rows, per + 4000, rng, dtype), _csr(b_rows, n, rng, dtype)
    names = _check(handle, oracle_mod, A, B, dtype, passes, planned=passes == 2)
    assert "win_spills" in names
    if passes == 1:
        assert _rows(names, "win_fill") == m, names
    else:
        assert _rows(names, "win_count") == m, names
        # (rows of more columns than the CTA bin's are not window rows)
        assert _rows(names, "win_fill") >= m - (off.size if kind in ("wider", "more") else 0), names


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("columns", [9, 16, 17, 60])
def test_thread_per_row(handle, oracle_mod, columns, passes, dtype):
    """70,000 rows of up to 81 products on 9 columns; every 61st row that is not
    sampled has 81 products on `columns` columns."""
    rng = np.random.default_rng(columns)
    m, groups, n = 70_000, 500, 30_000
    b_rows = []  # per group 27 rows of 3 of the group's 9 columns
    for g in range(groups):
        base = int(rng.integers(0, n - 64))
        for k in range(27):
            b_rows.append(base + np.sort((np.arange(3) * 3 + rng.integers(0, 3, 3) + k % 9) % 9))
    first = len(b_rows)
    for g in range(groups):  # and 27 of 3 of `columns` columns, all of them used
        base = int(rng.integers(0, n - 64))
        for k in range(27):
            c = {(3 * k + j) % columns for j in range(3)}
            b_rows.append(base + np.array(sorted(c)))
    a_rows = []
    for r in range(m):
        g = int(rng.integers(groups))
        size = 27 if r % 3 else int(rng.integers(18, 28))
        a_rows.append(27 * g + np.sort(rng.choice(27, size, replace=False)))
    off = _unsampled(m, 61)
    for r in off:
        a_rows[r] = first + 27 * int(rng.integers(groups)) + np.arange(27)
    assert off.size > 500
    A, B = _csr(a_rows, len(b_rows), rng, dtype), _csr(b_rows, n, rng, dtype)
    names = _check(handle, oracle_mod, A, B, dtype, passes, planned=passes == 2)
    # one pass: rows by products, all in one bin; two: by columns
    assert names.get("thread_fill", 0) == (m if passes == 1 or columns <= 12 else m - off.size), names
