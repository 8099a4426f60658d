"""The stacked operands of a batch at the edges of the runs they are copied in
(128 or 512 positions) and of the 32-way search for a run's pair: pairs that end
at, before and after a run, empty pairs between them, more pairs than one or two
steps of the search tell apart."""
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


def _exact(rows, n):
    """rows x 9, n entries, the first rows full."""
    col = np.concatenate([np.arange(min(9, max(0, n - 9 * r))) for r in range(rows)])
    rpt = np.minimum(9 * np.arange(rows + 1), n).astype(np.int32)
    return brm.CSR(rows, 9, rpt, col.astype(np.int32), np.arange(1.0, n + 1))


def _check(ctx, oracle_mod, pairs):
    dev = [(brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)) for A, B in pairs]
    want = [oracle_mod.precise(A, B) for A, B in pairs]
    for i, C in enumerate(ctx.batch_precise(dev)):
        assert_same_csr(C.to_host(), want[i], f"batch pair {i}")
    pipe = ctx.batch_pipe(dev)
    try:
        for i, C in enumerate(pipe.run(dev)):
            assert_same_csr(C.to_host(), want[i], f"pipe pair {i}")
    finally:
        pipe.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("sizes", [
    [1], [0, 1, 0], [127], [128], [129], [511, 1, 512, 0, 0, 513],
    [128, 128, 128, 0, 129, 127, 1, 0], [3] * 31, [3] * 32, [5, 0] * 17, [2, 1, 0] * 342 + [700]])
def test_stack_edges(ctx, oracle_mod, sizes, dtype):
    B = brm.gen_uniform(9, 40, 5, seed=1).astype(dtype)
    # rows of a pair end at run edges too: as many rows as entries, or a ninth
    pairs = [(_exact(max(1, n if i % 2 else -(-n // 9)), n).astype(dtype), B) for i, n in enumerate(sizes)]
    _check(ctx, oracle_mod, pairs)


def test_stack_long_runs(ctx, oracle_mod):
    """Entries enough for runs of 512 (11 M of A), pairs of uneven sizes."""
    D = brm.gen_uniform(40_000, 40_000, 90, seed=2)
    I = brm.CSR(40_000, 40_000, np.arange(40_001, dtype=np.int32),
                np.arange(40_000, dtype=np.int32), np.ones(40_000))
    S = brm.gen_er(333, 4, seed=3)
    pairs = [(D, I), (S, S), (D, I), (S, S), (D, I)]
    dev = [(brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)) for A, B in pairs]
    for (A, _), C in zip(pairs, ctx.batch_precise(dev)):
        assert_same_csr(C.to_host(), A if A is D else oracle_mod.precise(S, S), "long runs")
