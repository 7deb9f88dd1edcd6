"""GPU: the split of a batch's C into its products (row pointers from 0, local
columns), at the edges of the split's chunks: products of 0 rows, without
entries, of one entry, next to products of several 4,096-entry and 2,048-row
chunks.  The structure and the values of these one-entry-per-row operands are
known in closed form, so the comparison is exact."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR

pytestmark = pytest.mark.gpu


def _banded(m: int, width: int, seed: int) -> tuple[HostCSR, HostCSR]:
    """A = a diagonal, B = `width` consecutive columns per row (clipped)."""
    rng = np.random.default_rng(seed)
    n = max(m, width)
    diag = HostCSR(m, m, np.arange(m + 1, dtype=np.int32), np.arange(m, dtype=np.int32),
                   rng.uniform(0.5, 1.0, m))
    first = np.minimum(np.arange(m), n - width)
    col = (first[:, None] + np.arange(width)[None, :]).astype(np.int32).ravel()
    rpt = (np.arange(m + 1) * width).astype(np.int32)
    return diag, HostCSR(m, n, rpt, col, rng.uniform(0.5, 1.0, m * width))


@pytest.mark.parametrize("sizes", [
    [(4096, 1)],
    [(1, 1), (4095, 1), (1, 1), (4097, 1)],
    [(0, 1), (5, 0), (0, 3), (2049, 4), (0, 1), (3, 2048), (7, 0)],
    [(1, 1)] * 40 + [(2048, 9)] + [(1, 3)] * 33,
    [(0, 1), (0, 1)],
])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_batch_split_edges(handle, sizes, dtype):
    from gpuspgemm_b200.api import DeviceCSR, batch, pack_batch
    pairs = [tuple(x.astype(dtype) for x in _banded(m, w, 7 + i))
             for i, (m, w) in enumerate(sizes)]
    pb = pack_batch([(DeviceCSR.from_host(a), DeviceCSR.from_host(b)) for a, b in pairs])
    out = batch(pb, handle)
    assert len(out) == len(pairs)
    for (a, b), c in zip(pairs, out):
        c = c.to_host()
        assert (c.m, c.n) == (a.m, b.n)
        assert np.array_equal(c.rpt, b.rpt) and np.array_equal(c.col, b.col)
        assert np.array_equal(c.val, np.repeat(a.val, np.diff(b.rpt)) * b.val)
