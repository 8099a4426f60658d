"""Rank rows (at most 64 lists, placed by population counts): rows at the edges
of every class -- products, lists, column range, columns of one product and
columns shared by most lists, empty lists between the others -- against the
oracle, bit for bit, through every form and value type."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu

# (products, lists, empty lists) around the limits of the classes
EDGES = [(33, 2, 0), (64, 3, 1), (127, 32, 0), (128, 5, 3), (129, 32, 0), (383, 31, 1), (384, 7, 0),
         (385, 20, 12), (767, 32, 0), (768, 32, 0), (769, 9, 0), (1536, 32, 0), (1537, 17, 2),
         (3072, 32, 0), (3073, 30, 2), (6144, 32, 0), (6145, 32, 0), (5888, 21, 0),
         (128, 33, 0), (129, 33, 0), (500, 40, 24), (129, 65, 0), (700, 300, 9), (3072, 70, 0), (3000, 2000, 5), (768, 64, 0), (769, 64, 0), (2000, 48, 16),
         (3072, 64, 0), (3073, 64, 0), (600, 65, 0)]


def edge_rows(ncols, seed, repeats=0):
    """A, B: one A row per edge, each with B rows of its own whose lengths add
    up to the row's products, columns within [0, ncols) reaching both ends."""
    rng = np.random.default_rng(seed)
    a_rpt, b_rpt, b_col, nb = [0], [0], [], 0
    for products, lists, empty in EDGES:
        lists = max(lists, -(-products // ncols))  # a list holds a column once
        cuts = np.sort(rng.choice(products - 1, lists - 1, replace=False)) + 1
        lens = np.diff(np.concatenate([[0], cuts, [products]]))
        while lens.max() > ncols:  # lists longer than the range: even lengths
            lens = np.full(lists, products // lists) + (np.arange(lists) < products % lists)
        lens = np.concatenate([lens, np.zeros(empty, int)])
        rng.shuffle(lens)
        for i, n in enumerate(lens):
            c = np.sort(rng.choice(ncols, n, replace=False))
            if n and ncols > 2 and i == np.flatnonzero(lens)[0]:
                c[0], c[-1] = (0, ncols - 1) if n > 1 else (0, 0)
            if n > 2 and repeats:
                c[1] = c[0]
            b_col.append(c)
            b_rpt.append(b_rpt[-1] + n)
        nb += len(lens)
        a_rpt.append(nb)
    b_col = np.concatenate(b_col)
    A = brm.CSR(len(EDGES), nb, np.array(a_rpt, np.int32), np.arange(nb, dtype=np.int32),
                rng.uniform(-1, 1, nb))
    B = brm.CSR(nb, ncols, np.array(b_rpt, np.int32), b_col.astype(np.int32),
                rng.uniform(-1, 1, len(b_col)))
    return A, B


@pytest.fixture(scope="module")
def ctx():
    import torch  # noqa: F401
    c = brm.Context()
    yield c
    c.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("ncols", [250, 4096, 49153, 1 << 18, (1 << 18) + 1, 1 << 19,
                                   (1 << 19) + 1, 1 << 21])
def test_edges(ctx, oracle_mod, ncols, dtype):
    A, B = (X.astype(dtype) for X in edge_rows(ncols, seed=ncols))
    R = oracle_mod.precise(A, B)
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, "one call")
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")


def test_many_short_rows(ctx, oracle_mod):
    """Enough rows that they are claimed several at a time."""
    A = brm.gen_uniform(60000, 500, 13, seed=1)
    B = brm.gen_uniform(500, 9000, 30, seed=2)
    R = oracle_mod.precise(A, B)
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.precise_device(dA, dB).to_host(), R, "one call")
    assert_same_csr(ctx.precise(dA, dB).to_host(), R, "split")


@pytest.mark.parametrize("ncols", [300, 4096, 1 << 18])
def test_repeated_columns_are_summed(ctx, ncols):
    """B rows that repeat a column (not valid CSR, and refused when inputs are
    checked) are summed all the same; whole numbers make the sums exact."""
    A, B = edge_rows(ncols, seed=7 + ncols, repeats=1)
    keep = np.array([p <= 3072 and k <= 64 for p, k, _ in EDGES])
    A.val, B.val = np.rint(A.val * 8), np.rint(B.val * 8)
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    with pytest.raises(brm.BrmError):
        brm.brmerge_precise(A, B)
    R = A.to_scipy() @ B.to_scipy()
    for C in (ctx.precise(dA, dB), ctx.precise_device(dA, dB)):
        C = C.to_host()
        for row in np.flatnonzero(keep):
            s, e = C.rpt[row], C.rpt[row + 1]
            dense = np.zeros(ncols)
            dense[C.col[s:e]] = C.val[s:e]
            assert np.all(np.diff(C.col[s:e]) > 0)
            assert np.array_equal(dense, np.asarray(R[row].todense()).ravel()), row
