"""What a call leaves allocated in the device's memory pool once its results are
released: a batch's stacked operands go back with the call, when it fails too;
and what a small result keeps: at most twice its size, or 8 MiB more."""
import ctypes as C
import gc

import numpy as np
import pytest

import brmerge_gb300 as brm

pytestmark = pytest.mark.gpu


def pool_used():
    """Bytes in use in the current device's default pool (driver API)."""
    import torch
    torch.cuda.synchronize()
    gc.collect()
    cu = C.CDLL("libcuda.so.1")
    pool, used = C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # USED_MEM_CURRENT
    return used.value


def test_stacked_operands_go_back():
    import torch
    ctx = brm.Context()
    # 16 rows of A use 4 rows of a B of 96 MB, twice: 192 MB stacked, 10240 products
    rows, per = 100_000, 80
    rpt = torch.arange(rows + 1, device="cuda", dtype=torch.int32) * per
    col = torch.arange(per, device="cuda", dtype=torch.int32).repeat(rows)
    B = brm.DeviceCSR(rows, per, rpt, col, torch.ones(rows * per, device="cuda", dtype=torch.float64))
    A = brm.CSR(16, rows, np.arange(17, dtype=np.int32) * 4,
                np.tile(np.arange(4, dtype=np.int32), 16), np.ones(64))
    bad = brm.CSR(16, rows, A.rpt, A.col.copy(), A.val)
    bad.col[63] = 2 * rows + 5
    dA, dbad = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(bad)
    before = pool_used()
    res = ctx.batch_precise([(dA, B), (dA, B)])
    assert float(res[1].val.sum()) == 16 * 4 * per
    del res
    assert pool_used() - before < 64 << 20
    with pytest.raises(brm.BrmError):
        ctx.batch_precise([(dA, B), (dbad, B)])
    assert pool_used() - before < 64 << 20
    ctx.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [4, 12, 14])  # 27-point stencil: up to 729 products for 125 entries
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
    assert pool_used() - before <= 4 * (A.M + 1) + max(2 * size, size + (8 << 20)) + 4096
    assert np.array_equal(C_.to_host().val, R.val) and np.array_equal(C_.to_host().col, R.col)
    ctx.close()
