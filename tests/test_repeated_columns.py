"""B rows that repeat one column many times (not valid CSR; inputs unchecked):
the rank rows and the rows of the segment kernel add every product, however
many there are.  Whole numbers make the sums exact in any order."""
import numpy as np
import pytest

import brmerge_gb300 as brm

pytestmark = pytest.mark.gpu


def operands(lists, per, repeats, ncols, seed=3):
    """One A row; every B row holds column 11, the middle one `repeats` times."""
    rng = np.random.default_rng(seed)
    cols = []
    for i in range(lists):
        others = rng.choice(ncols - 12, per - 1, replace=False) + 12
        cols.append(np.sort(np.r_[others, [11] * (repeats if i == lists // 2 else 1)]))
    rpt = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    A = brm.CSR(1, lists, np.array([0, lists], np.int32), np.arange(lists, dtype=np.int32),
                rng.integers(-8, 9, lists).astype(float))
    B = brm.CSR(lists, ncols, rpt.astype(np.int32), np.concatenate(cols).astype(np.int32),
                rng.integers(-8, 9, rpt[-1]).astype(float))
    return A, B


@pytest.mark.parametrize("lists,per,repeats", [
    (5, 3, 20), (5, 3, 60), (5, 3, 100),           # at most 128 products
    (10, 12, 40), (10, 12, 63), (10, 12, 90), (10, 12, 200),  # by rank, one warp
    (30, 60, 300), (50, 40, 100),                  # more warps, two mask words a column
    (100, 5, 8), (100, 5, 16), (100, 5, 40), (200, 6, 900)])  # the segment kernel
def test_every_product_is_added(lists, per, repeats):
    ncols = 4000
    A, B = operands(lists, per, repeats, ncols)
    want = np.zeros(ncols)
    for j in range(lists):
        s, e = B.rpt[j], B.rpt[j + 1]
        np.add.at(want, B.col[s:e], A.val[j] * B.val[s:e])
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    for C in (ctx.precise(dA, dB), ctx.precise_device(dA, dB), ctx.upper(dA, dB)):
        C = C.to_host()
        assert np.all(np.diff(C.col) > 0)
        got = np.zeros(ncols)
        got[C.col] = C.val
        assert np.array_equal(got, want)
    ctx.close()
