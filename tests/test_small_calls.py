"""Small one-call products: the offset scan at the edges of its tiles and of its
one-launch form, calls on both sides of the size from which nnz(C) is waited
for before C is allocated, few rows of several rank classes in one launch, and
a call that fails without having waited."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch  # noqa: F401
    c = brm.Context()
    yield c
    c.close()


def check(ctx, oracle_mod, A, B, what):
    R = oracle_mod.precise(A, B)
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, what + " one call")
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, what + " split")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, what + " upper")


@pytest.mark.parametrize("rows", [1, 4095, 4096, 4097, 32768, 32769, 70001])
def test_scan_tiles(ctx, oracle_mod, rows):
    A = brm.gen_uniform(rows, 300, 4, seed=rows)
    check(ctx, oracle_mod, A, brm.gen_uniform(300, 500, 12, seed=3), str(rows))


@pytest.mark.parametrize("n", [32767, 32768, 32769])  # 64 products a row, 2^21 at 32768 rows
def test_waiting_for_nnz(ctx, oracle_mod, n):
    A = brm.gen_er(n, 8, seed=n)
    check(ctx, oracle_mod, A, A, str(n))


@pytest.mark.parametrize("rows", [1, 5, 60, 300, 1200, 4000])
def test_few_rows_of_many_classes(ctx, oracle_mod, rows):
    """From a few to a few thousand products a row (the rank classes of at most
    32 lists), copy, warp and empty rows among them."""
    B = brm.gen_lognormal(2000, 3000, mu=3.5, sigma=1.2, cap=400, seed=5)
    check(ctx, oracle_mod, brm.gen_uniform(rows, 2000, 30, seed=rows), B, str(rows))


def test_failed_call(ctx, oracle_mod):
    A = brm.gen_er(500, 6, seed=1)
    bad = A.copy()
    bad.col[bad.rpt[250] + 5] = 500  # a column without a row of B
    dA, dbad = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(bad)
    for _ in range(2):
        with pytest.raises(brm.BrmError) as e:
            ctx.precise_device(dbad, dA)
        assert e.value.status == 2  # BRM_ERR_INVALID_CSR
        check(ctx, oracle_mod, A, A, "after a failure")
    # new values on the plan of a call that did not wait
    C = ctx.precise_device(dA, dA)
    A2 = brm.CSR(A.M, A.N, A.rpt, A.col, A.val * 3)
    dA.val.copy_(brm.DeviceCSR.from_host(A2).val)
    C2 = ctx.numeric(dA, dA, C.rpt, int(C.rpt[-1]))
    assert_same_csr(C2.to_host(), oracle_mod.precise(A2, A2), "numeric after one call")
