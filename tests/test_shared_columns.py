"""Rows of 3073 to 5888 products and 33 to 255 lists: merged by a group of warps
where the column range holds at most a third as many columns as the row has
products (and a thread's share is not 32 products) and the matrix has 2048 rows or
more than 32 entries a row, cut into segments elsewhere; both sides of every line, against the oracle, bit for
bit."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from brmerge_gb300 import _native
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu

# lists, products, columns, merged
ROWS = [(60, 3600, 1200, True), (60, 3600, 1201, False), (33, 3073, 1024, True),
        (33, 3073, 1025, False), (255, 3073, 40, True), (255, 5888, 1962, True),
        (255, 5888, 1963, False), (255, 5889, 300, False), (62, 3968, 500, True),
        (62, 3969, 500, False), (64, 4096, 500, False), (64, 4097, 500, True),
        (100, 5000, 401, True), (200, 4600, 100000, False)]


def one_row(lists, products, ncols, dtype, seed, rows=2048):
    """A of one row (and empty ones) with a B row of its own for each entry; the
    first and the last column are used."""
    rng = np.random.default_rng(seed)
    lens = np.full(lists, products // lists) + (np.arange(lists) < products % lists)
    cols = [np.sort(rng.choice(ncols, n, replace=False)) for n in lens]
    cols[0][0], cols[0][-1] = 0, ncols - 1
    rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    a_rpt = np.full(rows + 1, lists, np.int32)
    a_rpt[0] = 0
    A = brm.CSR(rows, lists, a_rpt, np.arange(lists, dtype=np.int32), rng.uniform(-1, 1, lists))
    B = brm.CSR(lists, ncols, rpt, np.concatenate(cols).astype(np.int32),
                rng.uniform(-1, 1, products))
    return A.astype(dtype), B.astype(dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("lists,products,ncols,merged", ROWS)
def test_both_routes(oracle_mod, lists, products, ncols, merged, dtype):
    A, B = one_row(lists, products, ncols, dtype, seed=products)
    R = oracle_mod.precise(A, B)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    before = _native.lib().brm_kernel_launches()
    C = ctx.precise_device(dA, dB)
    launches = _native.lib().brm_kernel_launches() - before
    assert_same_csr(C.to_host(), R, "one call")
    # merged: analysis, merge, scan, compaction; cut: planning and four more
    assert (launches <= 4) == merged, launches
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")
    ctx.close()


@pytest.mark.parametrize("rows,merged", [(2047, False), (2, False), (1, True)])
def test_few_rows(oracle_mod, rows, merged):
    A, B = one_row(60, 3600, 1200, np.float64, seed=1, rows=rows)
    R = oracle_mod.precise(A, B)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    before = _native.lib().brm_kernel_launches()
    C = ctx.precise_device(dA, dB)
    assert (_native.lib().brm_kernel_launches() - before <= 4) == merged
    assert_same_csr(C.to_host(), R, "one call")
    ctx.close()
