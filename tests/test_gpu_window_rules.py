"""GPU: where the window and thread-per-row kernels stop, on both sides of each
rule: the span in words per product, words and columns of four-lane teams, B rows
too short for a team, and the thread-per-row fill whatever the span.  Against the
oracle: structure bit-exact, values within 1e-12 of sum |a||b|."""
import numpy as np
import pytest

from gpuspgemm_b200.csr import HostCSR
from test_gpu_window_dispatch import _check, _rows

pytestmark = pytest.mark.gpu


def _even(m, a_len, b_len, width, stretch, seed=3):
    """m rows of a_len B rows of b_len entries; a row's columns fall evenly on
    `width` columns, `stretch` apart."""
    rng = np.random.default_rng(seed)
    groups, per = 10, 8 * a_len
    j = np.arange(b_len)
    lo, hi = j * width // b_len, (j + 1) * width // b_len
    col = lo + rng.integers(0, 1 << 30, (groups * per, b_len)) % (hi - lo)
    col = (col + np.arange(groups).repeat(per)[:, None] * width) * stretch
    b_rpt = np.arange(groups * per + 1, dtype=np.int32) * b_len
    B = HostCSR(groups * per, groups * width * stretch, b_rpt, col.astype(np.int32).ravel(),
                rng.uniform(-1, 1, col.size))
    acol = (rng.integers(0, groups, (m, 1)) * per + np.arange(a_len) * 8 +
            rng.integers(0, 8, (m, a_len)))
    A = HostCSR(m, groups * per, np.arange(m + 1, dtype=np.int32) * a_len,
                acol.astype(np.int32).ravel(), rng.uniform(-1, 1, acol.size))
    return A, B


# words (of the sampled span and a tenth more) per product: one pass up to 2.0,
# two passes' count 1.65, their fill 1.5, times the share of the team's lanes
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("stretch,count,fill", [(1, True, True), (64, True, True),
                                                (120, True, False), (144, False, False),
                                                (256, False, False)])
def test_span(handle, oracle_mod, stretch, count, fill, passes):
    a_len, b_len, width = 20, 15, 107  # 300 products, 15 of 16 lanes
    A, B = _even(4000, a_len, b_len, width, stretch)
    words = 1.1 * width * stretch / 32 / (a_len * b_len) / (b_len / 16)
    assert (words < 1.65) == count and (words < 1.5) == fill
    names = _check(handle, oracle_mod, A, B, np.float64, passes, planned=passes == 2)
    if passes == 1:
        assert (_rows(names, "win_fill") > 0) == (words < 2.0), names
    else:
        assert (_rows(names, "win_count") > 0) == count, names
        assert (_rows(names, "win_fill") > 0) == fill, names


@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("b_len,a_len,width,stretch,windows",
                         [(3, 40, 30, 1, True), (3, 60, 60, 1, False),    # columns held
                          (4, 40, 14, 100, True), (4, 40, 14, 512, False),  # words a lane
                          (2, 60, 24, 1, None), (3, 40, 24, 1, True)])      # short B rows
def test_four_lanes(handle, oracle_mod, b_len, a_len, width, stretch, windows, passes):
    A, B = _even(6000, a_len, b_len, width, stretch)
    names = _check(handle, oracle_mod, A, B, np.float64, passes, planned=passes == 2)
    # (B rows of two: only the fill of two passes stays away)
    want = passes == 1 if windows is None else windows
    assert (_rows(names, "win_fill4") > 0) == want, names


@pytest.mark.parametrize("stretch", [1, 256])
def test_thread_per_row_at_any_span(handle, oracle_mod, stretch):
    A, B = _even(70_000, 27, 3, 9, stretch)
    for passes in (1, 2):
        names = _check(handle, oracle_mod, A, B, np.float64, passes, planned=passes == 2)
        assert names.get("thread_fill") == 70_000, names
