"""Long columns of heavy rows (more than 32 products) in a scratch of every size,
from one that holds none of them to one that its records just fit: each product
of the row in one of a few columns, so that the columns fill the scratch."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_column", [33, 34, 64])
def test_scratch_of_every_size(oracle_mod, per_column):
    rng = np.random.default_rng(per_column)
    lists, per = 400, 150  # 60000 products a row: heavy
    ncols = lists * per // per_column
    cols = [np.sort((lst + lists * np.arange(per)) % ncols) for lst in range(lists)]
    rpt = np.arange(lists + 1, dtype=np.int32) * per
    B = brm.CSR(lists, ncols, rpt, np.concatenate(cols).astype(np.int32),
                rng.uniform(-1, 1, rpt[-1]))
    A = brm.CSR(3, lists, np.arange(4, dtype=np.int32) * lists,
                np.tile(np.arange(lists, dtype=np.int32), 3), rng.uniform(-1, 1, 3 * lists))
    R = oracle_mod.precise(A, B)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    for scratch in (1, 33, 1000, 3 * int(rpt[-1]) - 1, 3 * int(rpt[-1]), None):
        ctx.set_tuning(long_scratch=scratch) if scratch else ctx.set_tuning()
        assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, f"one call, scratch {scratch}")
        assert_same_csr(ctx.upper(dA, dB).to_host(), R, f"upper, scratch {scratch}")
    ctx.close()
