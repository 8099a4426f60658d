"""Rank rows at the lines that the column range draws: short rows on both sides
of the range at which they have a pack to themselves (many and few of them, few
and many lists), rows of 33 to 64 lists whose columns are as many as their
products, one fewer and one more, rows of 3073 to 3969 products that reach into a
second planning chunk.  Against the oracle, bit for bit."""
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
    cols = list(cols) + [np.zeros(0, np.int64)] * (rows - len(cols))  # empty rows
    rpt = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return brm.CSR(rows, ncols, rpt, np.concatenate(cols).astype(np.int32),
                   rng.uniform(-1, 1, rpt[-1])).astype(dtype)


def spread(ncols, n, rng):
    """n sorted distinct columns, the first and the last one among them."""
    inner = rng.choice(ncols - 2, n - 2, replace=False) + 1 if n > 2 else []
    return np.sort(np.r_[0, inner, ncols - 1][:n]).astype(np.int64)


@pytest.mark.parametrize("rows", [3, 16383, 16384])
@pytest.mark.parametrize("ncols", [1 << 16, (1 << 16) + 1025, 1 << 17, (1 << 17) + 1, 1 << 18,
                                   (1 << 18) + 1])
def test_short_rows(oracle_mod, ncols, rows):
    """2 to 128 products of 2 to 32 lists, every row over all of the range."""
    rng = np.random.default_rng(ncols)
    lens = [2, 3, 4, 8, 16, 30, 31, 32]
    B = csr(256, ncols, [spread(ncols, lens[i % 8], rng) for i in range(256)], rng, np.float64)
    picks = [[0, 8], [5, 7], [7, 15], [0, 8, 16, 24, 32, 40, 48, 56], [1, 9, 17, 25, 33, 41, 49, 57, 65],
             [6, 14], [7, 15, 23, 31], [4, 12, 20, 28, 36], list(range(0, 128, 8)),
             list(range(0, 256, 8)), [3, 11, 19, 27], [7, 14]]
    picks = [sorted(picks[i % len(picks)]) for i in range(rows)]
    A = csr(rows, 256, [np.array(p) for p in picks], rng, np.float64)
    check(oracle_mod, A, B)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows", [4095, 4096])
@pytest.mark.parametrize("lists,products", [(33, 769), (64, 770), (40, 1600), (48, 2999), (64, 3072)])
def test_columns_as_many_as_products(oracle_mod, lists, products, rows, dtype):
    rng = np.random.default_rng(products)
    for ncols in (products - 1, products, products + 1, products + 2, 3 * products):
        lens = np.full(lists, products // lists) + (np.arange(lists) < products % lists)
        B = csr(lists, ncols, [spread(ncols, n, rng) for n in lens], rng, dtype)
        A = csr(rows, lists, [np.arange(lists)], rng, dtype)
        check(oracle_mod, A, B)


@pytest.mark.parametrize("products", [3073, 3968, 3969])
@pytest.mark.parametrize("ncols", [1 << 18, (1 << 18) + 1, 1 << 19])
def test_second_planning_chunk(oracle_mod, ncols, products):
    rng = np.random.default_rng(products)
    lens = np.full(40, products // 40) + (np.arange(40) < products % 40)
    B = csr(40, ncols, [spread(ncols, n, rng) for n in lens], rng, np.float64)
    for rows in (2047, 2048):
        check(oracle_mod, csr(rows, 40, [np.arange(40)], rng, np.float64), B)
