"""GPU: transpose at the edges of its kernels' ranges: columns of 1, 127-129,
2047-2049 and 16383-16385 entries beside empty ones, entry counts around a
warp's scatter tile (256) and one row holding many tiles.  Values are moved
without arithmetic, so the comparison is bit for bit."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu


def _columns(lengths, m, seed):
    """m x len(lengths), column j holding lengths[j] entries in random rows."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([rng.choice(m, size=k, replace=False) for k in lengths])
    cols = np.repeat(np.arange(len(lengths)), lengths)
    order = np.lexsort((cols, rows))
    rpt = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))])
    return HostCSR(m, len(lengths), rpt.astype(np.int32), cols[order].astype(np.int32),
                   rng.uniform(-1, 1, rows.size))


def _one_row(nnz, m, seed):
    """All entries in one row in the middle of m rows."""
    rpt = np.zeros(m + 1, np.int32)
    rpt[m // 2 + 1:] = nnz
    return HostCSR(m, nnz + 3, rpt, np.arange(nnz, dtype=np.int32) + 1,
                   np.random.default_rng(seed).uniform(-1, 1, nnz))


CASES = {
    "lengths": lambda: _columns([1, 0, 127, 128, 129, 0, 0, 2047, 2048, 2049, 16383, 16384,
                                 16385, 1], 20_000, 3),
    "short": lambda: _columns([3, 0, 1, 2] * 700, 40, 4),
    "dense128": lambda: _columns([128] * 37, 128, 5),
    "entries1": lambda: _one_row(1, 1, 6),
    "entries255": lambda: _one_row(255, 3, 7),
    "entries256": lambda: _one_row(256, 70, 8),
    "entries257": lambda: _one_row(257, 2, 9),
    "entries5000": lambda: _one_row(5000, 100_000, 10),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_transpose_edges(handle, oracle_mod, name, dtype):
    from gpuspgemm_b200.api import DeviceCSR, transpose
    A = CASES[name]().astype(dtype)
    T = transpose(DeviceCSR.from_host(A), handle).to_host()
    R = oracle_mod.transpose(A)
    assert (T.m, T.n) == (R.m, R.n)
    assert np.array_equal(T.rpt, R.rpt) and np.array_equal(T.col, R.col)
    assert np.array_equal(T.val, R.val)
