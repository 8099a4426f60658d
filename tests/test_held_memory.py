"""What calls leave allocated in the device's memory pool once their results are
released: a batch's stacked operands up to a bound, none of them in a server's
workers, after an error or after a pipeline's capacities were taken from a sample;
and what a small result keeps: at most twice its size, or 16 MiB more."""
import ctypes as C
import gc

import numpy as np
import pytest

import brmerge_gb300 as brm

pytestmark = pytest.mark.gpu


def pool_used():
    """Bytes in use in the current device's default pool (driver API); what a
    plain cudaFree gives back stays in this count."""
    import torch
    torch.cuda.synchronize()
    gc.collect()
    cu = C.CDLL("libcuda.so.1")
    pool, used = C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # USED_MEM_CURRENT
    return used.value


@pytest.fixture(scope="module")
def pair():
    """16 rows of A use 4 rows of a B of 96 MB: 5120 products."""
    import torch
    rows, per = 100_000, 80
    rpt = torch.arange(rows + 1, device="cuda", dtype=torch.int32) * per
    col = torch.arange(per, device="cuda", dtype=torch.int32).repeat(rows)
    B = brm.DeviceCSR(rows, per, rpt, col, torch.ones(rows * per, device="cuda", dtype=torch.float64))
    A = brm.CSR(16, rows, np.arange(17, dtype=np.int32) * 4,
                np.tile(np.arange(4, dtype=np.int32), 16), np.ones(64))
    bad = brm.CSR(16, rows, A.rpt, A.col.copy(), A.val)
    bad.col[63] = 100 * rows
    return brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(bad), B


SMALL = 64 << 20  # what else the context may hold here


def test_stacked_operands_of_a_context(pair):
    A, bad, B = pair
    before = pool_used()
    ctx = brm.Context()
    for n, kept in ((2, 192_000_000), (60, 0), (2, 192_000_000)):  # 5.8 GB: above the bound
        res = ctx.batch_precise([(A, B)] * n)
        assert float(res[-1].val.sum()) == 16 * 4 * 80
        del res
        assert 0 <= pool_used() - before - kept < SMALL, n
    with pytest.raises(brm.BrmError):
        ctx.batch_precise([(A, B), (bad, B)])
    assert pool_used() - before < SMALL
    ctx.batch_precise([(A, B)] * 2)
    held = pool_used()
    # (the pipeline's own pool buffers are 64 MiB of spill scratch and small ones)
    pipe = ctx.batch_pipe([(A, B)] * 2)
    assert pool_used() - held < -192_000_000 + (64 << 20) + SMALL
    pipe.close()
    ctx.close()


def test_stacked_operands_of_a_server(pair):
    A, _, B = pair
    before = pool_used()
    srv = brm.Server(workers=1)
    for t in [srv.submit(A, B) for _ in range(3)]:
        C_, _ = srv.wait(t, timeout=60.0)
        assert float(C_.val.sum()) == 16 * 4 * 80
        del C_
    assert pool_used() - before < SMALL
    srv.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [4, 12, 15])  # 27-point stencil: up to 729 products for 125 entries
def test_room_of_a_small_result(oracle_mod, n, dtype):
    A = brm.gen_stencil27(n).astype(dtype)
    R = oracle_mod.precise(A, A)
    ctx = brm.Context()
    dA = brm.DeviceCSR.from_host(A)
    C_ = ctx.precise_device(dA, dA)  # (the context's own buffers)
    del C_
    before = pool_used()
    C_ = ctx.precise_device(dA, dA)
    size = len(R.col) * (4 + R.val.itemsize)
    assert pool_used() - before <= 4 * (A.M + 1) + max(2 * size, size + (16 << 20)) + 4096
    assert np.array_equal(C_.to_host().val, R.val) and np.array_equal(C_.to_host().col, R.col)
    ctx.close()
