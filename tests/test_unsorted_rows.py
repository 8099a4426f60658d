"""Short rows whose B rows are not sorted, with columns outside their first and
last one (not valid CSR; inputs unchecked), multiplied all the same: rows of at
most 32 products in any order, rows of at most 128 products and 32 lists where
no column lies before the first ones.  On their own, among sorted rows and
beside a longer one.  The order of a column's additions depends on the list, not
on the place within it, so the result is the sorted operand's, bit for bit."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu


def operands(rows, ncols, most, longest, share, dtype, seed):
    """A: 2..32 entries a row, at most `most` products; B rows of 2..8 entries, a
    `share` of them shuffled.  longest: products of a last row by itself, its B
    rows sorted (0: none)."""
    rng = np.random.default_rng(seed)
    nb = 400
    lens = rng.integers(2, 9, nb)
    cols = [np.sort(rng.choice(ncols, n, replace=False)) for n in lens]
    a_cols = []
    for _ in range(rows):
        pick = rng.choice(nb, rng.integers(2, 33), replace=False)
        a_cols.append(np.sort(pick[:max(2, np.searchsorted(np.cumsum(lens[pick]), most, "right"))]))
    if longest:
        per = longest // 16
        cols += [np.sort(rng.choice(ncols, per, replace=False)) for _ in range(16)]
        a_cols.append(np.arange(nb, nb + 16))
    rpt = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    order = np.arange(rpt[-1])
    for i in range(nb):
        first = rpt[i] + (most > 32)
        if rng.random() < share:
            order[first:rpt[i + 1]] = rng.permutation(order[first:rpt[i + 1]])
    a_rpt = np.concatenate([[0], np.cumsum([len(c) for c in a_cols])]).astype(np.int32)
    A = brm.CSR(len(a_cols), len(cols), a_rpt, np.concatenate(a_cols).astype(np.int32),
                rng.uniform(-1, 1, a_rpt[-1])).astype(dtype)
    S = brm.CSR(len(cols), ncols, rpt, np.concatenate(cols).astype(np.int32),
                rng.uniform(-1, 1, rpt[-1])).astype(dtype)
    B = brm.CSR(S.M, S.N, rpt, S.col[order], S.val[order])
    return A, B, S


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("most", [32, 128])
@pytest.mark.parametrize("share", [0.05, 1.0])
@pytest.mark.parametrize("rows,ncols,longest", [(1, 900, 0), (7, 900, 0), (20000, 5000, 0),
                                                (20000, 1 << 17, 0), (200, 900, 320),
                                                (200, 5000, 640), (300, 1 << 17, 1280),
                                                (200, 5000, 2400), (100, 5000, 4800)])
def test_short_rows_in_any_order(oracle_mod, rows, ncols, longest, share, most, dtype):
    A, B, S = operands(rows, ncols, most, longest, share, dtype, seed=rows + longest)
    R = oracle_mod.precise(A, S)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, "one call")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")
    ctx.close()


def test_batches_in_any_order(oracle_mod):
    ctx = brm.Context()
    dev = []
    for i in range(5):
        A, B, S = operands(50, 700, 32, 0, i % 2, np.float64, seed=i)
        dev.append(((brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)),
                    oracle_mod.precise(A, S)))
    sorted_first = [p for p, _ in dev[::2]]
    pipe = ctx.batch_pipe([p for p, _ in dev])
    for _ in range(2):
        for what, run in (("batch", ctx.batch_precise), ("pipe", pipe.run)):
            for C, (_, R) in zip(run([p for p, _ in dev]), dev):
                assert_same_csr(C.to_host(), R, what)
            for C, (_, R) in zip(run(sorted_first), dev[::2]):
                assert_same_csr(C.to_host(), R, what + " sorted")
    pipe.close()
    ctx.close()
