"""GPU: products of more rows than the one-launch binning takes (2^22), whose rows
go through the three-launch binning and its kernels: the sort kernels that share a
row list by the row's size, with the split chosen by option and by the sample, B
up to 2^20 columns and past it; and the window and thread-per-row fills.  Most
rows are empty or hold one product; a few hundred, some of them at the sampled
places, have as many products as each kernel's limit, or one more or fewer.
Against the oracle: structure bit-exact, values within 1e-12 (FP64) or 1e-5 (FP32)
of sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu

M = (1 << 22) + 77
SAMPLED = (np.arange(2048, dtype=np.int64) * M) // 2048
SIZES = [2, 12, 13, 48, 49, 192, 193, 300, 400, 511, 512, 513, 640, 767, 768, 769, 1023, 1024, 1025,
         2047, 2048, 2049, 3071, 3072, 3073, 12288, 12289]


def _csr(rows, at, m, n, rng, dtype):
    """m rows, `rows[i]` at row at[i], the others empty."""
    order = np.argsort(at, kind="stable")
    lens = np.zeros(m, np.int64)
    lens[at] = [rows[i].size for i in range(len(rows))]
    rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([rows[i] for i in order]).astype(np.int32)
    return HostCSR(m, n, rpt, col, rng.uniform(-1, 1, col.size).astype(dtype))


def _positions(count, rng):
    """Places of `count` rows: a third of them sampled ones, with both ends of A."""
    own = np.concatenate([rng.choice(SAMPLED[1:], count // 3, replace=False), [0, M - 1]])
    rest = np.setdiff1d(rng.choice(M, 2 * count, replace=False), own)
    return np.concatenate([own, rng.permutation(rest)[:count - own.size]])


def _check(handle, oracle_mod, A, B, dtype, passes, esc=0):
    from gpuspgemm_b200 import _native as N
    from gpuspgemm_b200.api import DeviceCSR, proposal
    handle.set_option(N.OPT_ONE_PASS, passes)
    handle.set_option(N.OPT_ESC, esc)
    handle.set_option(N.OPT_PROFILE, 1)
    try:
        C = proposal(DeviceCSR.from_host(A), DeviceCSR.from_host(B), handle).to_host()
        names = {k["name"] for k in handle.profile()}
    finally:
        handle.set_option(N.OPT_PROFILE, 0)
        handle.set_option(N.OPT_ONE_PASS, 0)
        handle.set_option(N.OPT_ESC, 0)
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    R = oracle_mod.spgemm(A64, B64, np.float64)
    res = oracle_mod.compare(C, R, oracle_mod.abs_bound(A64, B64, R))
    assert res["rpt_equal"] and res["col_equal"], res
    assert res.get("max_cond", 0.0) <= (1e-12 if dtype == np.float64 else 1e-5), res
    return names


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("esc", [0, 1])
@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1, 1 << 22])
def test_sort_kernels(handle, oracle_mod, n, esc, dtype):
    rng = np.random.default_rng(n + esc)
    # B: 3,000 rows of one column, then 3,000 of 2 to 20, over all of B.n
    b_rows = [np.array([int(rng.integers(n))]) for _ in range(3000)]
    b_rows += [np.unique(rng.integers(0, n, int(rng.integers(2, 21)))) for _ in range(3000)]
    b_rows[0], b_rows[1] = np.array([0]), np.array([n - 1])
    lens = np.array([r.size for r in b_rows])
    B = _csr(b_rows, np.arange(6000), 6000, n, rng, dtype)
    a_rows = []
    for size in SIZES * 12:  # exactly `size` products
        pick = 3000 + rng.permutation(3000)
        cut = int(np.searchsorted(np.cumsum(lens[pick]), size, side="right"))
        left = size - int(lens[pick[:cut]].sum())
        ones = rng.choice(3000, min(left, 3000), replace=False)
        a_rows.append(np.sort(np.concatenate([pick[:cut], ones])))
    many = len(a_rows)
    a_rows += [np.array([int(rng.integers(6000))]) for _ in range(40_000)]
    at = _positions(many, rng)
    free = np.setdiff1d(rng.choice(M, 41_500, replace=False), np.concatenate([at, SAMPLED]))[:40_000]
    A = _csr(a_rows, np.concatenate([at, free]), M, 6000, rng, dtype)
    assert A.nnz > 1 << 15
    names = _check(handle, oracle_mod, A, B, dtype, 1, esc)
    # the split at 512 products, and the list that two kernels share
    assert {"esc_team32_n512", "esc_cta256_n3072"} <= names, names
    if n > 1 << 20:
        assert {"esc_cta1024_n12288", "s2n_bitmap1024_ranges"} <= names, names


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("passes", [1, 2])
def test_window_kernels(handle, oracle_mod, passes, dtype):
    rng = np.random.default_rng(passes)
    n, per = 50_000, 60
    # 20 windows of 190 columns, 60 B rows of about 15 columns in each
    b_rows = []
    for g in range(20):
        base = int(rng.integers(0, n - 190))
        b_rows += [base + np.sort(rng.choice(190, int(rng.integers(8, 23)), replace=False))
                   for _ in range(per)]
    B = _csr(b_rows, np.arange(len(b_rows)), len(b_rows), n, rng, dtype)
    a_rows = [int(rng.integers(20)) * per + np.sort(rng.choice(per, int(rng.integers(20, 50)),
                                                               replace=False)) for _ in range(3000)]
    A = _csr(a_rows, _positions(3000, rng), M, len(b_rows), rng, dtype)
    names = _check(handle, oracle_mod, A, B, dtype, passes)
    assert any(x.startswith("win_fill") for x in names), names
    assert passes == 1 or any(x.startswith("win_count") for x in names), names
