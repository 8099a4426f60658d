"""Rank rows at the lines that the column range draws: rows of 33 to 64 lists
whose columns are as many as their products, one fewer and one more.  Against
the oracle, bit for bit."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu


def check(oracle_mod, A, B):
    R = oracle_mod.precise(A, B)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, "one call")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")
    ctx.close()


def csr(rows, ncols, cols, rng, dtype):
    rpt = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return brm.CSR(rows, ncols, rpt, np.concatenate(cols).astype(np.int32),
                   rng.uniform(-1, 1, rpt[-1])).astype(dtype)


def spread(ncols, n, rng):
    """n sorted distinct columns, the first and the last one among them."""
    inner = rng.choice(ncols - 2, n - 2, replace=False) + 1 if n > 2 else []
    return np.sort(np.r_[0, inner, ncols - 1][:n]).astype(np.int64)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("lists,products", [(33, 769), (64, 770), (40, 1600), (48, 2999), (64, 3072)])
def test_columns_as_many_as_products(oracle_mod, lists, products, dtype):
    rng = np.random.default_rng(products)
    for ncols in (products - 1, products, products + 1, products + 2, 3 * products):
        lens = np.full(lists, products // lists) + (np.arange(lists) < products % lists)
        B = csr(lists, ncols, [spread(ncols, n, rng) for n in lens], rng, dtype)
        A = csr(1, lists, [np.arange(lists)], rng, dtype)
        check(oracle_mod, A, B)
