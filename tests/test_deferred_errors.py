"""A small one-call product that does not wait for nnz(C) still reports what
its plan's kernels found: a B row that is not sorted, whose inner column lies
outside the row's first and last one, so that only the kernels of the row's
class see it (and skip it)."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu

NCOLS = 1 << 20


def operands(rows, seed=1):
    """A, B: one A row per (lists, products a list, first, last column, bad), with
    B rows of its own; bad: a column beyond the last in the middle of one."""
    rng = np.random.default_rng(seed)
    a_rpt, b_rpt, b_col = [0], [0], []
    for lists, per, lo, hi, bad in rows:
        for i in range(lists):
            c = np.sort(rng.choice(hi - lo - 1, per - 2, replace=False)) + lo + 1
            c = np.concatenate([[lo], c, [hi]])
            if bad and i == lists // 2:
                c[per // 2] = hi + 7
            b_col.append(c)
            b_rpt.append(b_rpt[-1] + per)
        a_rpt.append(a_rpt[-1] + lists)
    nb, b_col = len(b_rpt) - 1, np.concatenate(b_col)
    A = brm.CSR(len(rows), nb, np.array(a_rpt, np.int32), np.arange(nb, dtype=np.int32),
                rng.uniform(-1, 1, nb))
    B = brm.CSR(nb, NCOLS, np.array(b_rpt, np.int32), b_col.astype(np.int32),
                rng.uniform(-1, 1, len(b_col)))
    return A, B


BATCH = (100, 5, 0, NCOLS - 20, False)  # too wide for the rank and merge kernels: a batched row


@pytest.mark.parametrize("with_batch", [False, True])
@pytest.mark.parametrize("bad", [(20, 10, 500, 9000, True),     # by rank, one warp
                                 (20, 30, 500, 300000, True),   # by rank, four warps
                                 (40, 40, 500, 9000, True),     # two mask words a column
                                 (100, 5, 500, 9000, True)])    # a segment's kernel
def test_error_of_a_call_that_did_not_wait(oracle_mod, bad, with_batch):
    ctx = brm.Context()
    rows = [bad] + [BATCH] * with_batch
    dA, dB = (brm.DeviceCSR.from_host(X) for X in operands(rows))
    good = [brm.DeviceCSR.from_host(X) for X in operands([r[:4] + (False,) for r in rows])]
    R = oracle_mod.precise(*(X.to_host() for X in good))
    for _ in range(2):
        with pytest.raises(brm.BrmError) as e:
            ctx.precise_device(dA, dB)
        assert e.value.status == 2  # BRM_ERR_INVALID_CSR
        assert_same_csr(ctx.precise_device(*good).to_host(), R, "after a failure")
    ctx.close()
