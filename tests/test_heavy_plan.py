"""Planning of the heavy rows at the edges of its windows (4096 products, 512
lists at a time): empty lists, lists across windows, one long list, cuts where a
group of columns holds more products than a segment, more columns than a chunk."""
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


def _operands(lens, ncols, seed):
    """One row of A over all rows of B, whose lengths are lens."""
    rng = np.random.default_rng(seed)
    rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(ncols, n, replace=False)) for n in lens])
    B = brm.CSR(len(lens), ncols, rpt, col.astype(np.int32), rng.standard_normal(rpt[-1]))
    k = len(lens)
    A = brm.CSR(1, k, np.array([0, k], np.int32), np.arange(k, dtype=np.int32),
                rng.standard_normal(k))
    return A, B


@pytest.mark.parametrize("lens, ncols", [
    ([0, 8] * 256, 5000),                       # 512 lists, half of them empty
    ([8] * 511 + [9], 5000),                    # one product beyond a window
    ([8] * 511 + [7], 5000),                    # one short of it
    ([16] * 513, 300_000),                      # a second round of lists, two chunks
    ([1] * 255 + [0] * 257 + [9000] + [3] * 40, 200_000),
    ([4096] * 3, 70_000), ([4095, 1, 4097], 70_000), ([0, 0, 20_000, 1], 600_000),
    ([100] * 700, 128),                         # one group of columns, far above a segment
    ([60] * 300 + [2000] * 4, 4096)])
def test_plan_windows(ctx, oracle_mod, lens, ncols):
    A, B = _operands(lens, ncols, len(lens))
    R = oracle_mod.precise(A, B)
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, "one call")
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")
