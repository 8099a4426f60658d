"""Upper's compaction works in tiles of 4096 entries of C: row lengths that
end, start and stretch at the edges of tiles, empty rows between them."""
import numpy as np
import pytest

import brmerge_gb300 as brm
from conftest import assert_same_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [
    [4095], [4096], [4097], [1] * 4096, [1] * 4097, [4096, 1], [0, 0, 4096, 0, 1, 0],
    [20000, 3, 0, 9000] + [0] * 5000 + [7, 8192, 1], [0] * 300 + [1] + [0] * 70000 + [5],
    [2, 0, 1] * 30000], ids=lambda x: f"{len(x)}rows_{sum(x)}")
def test_tiles(oracle_mod, lens):
    rng = np.random.default_rng(len(lens))
    ncols = 50000
    rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(ncols, n, replace=False)) if n else []
                          for n in lens]).astype(np.int32)
    B = brm.CSR(len(lens), ncols, rpt, col, rng.uniform(-1, 1, len(col)))
    n = len(lens)
    # row i: B row i, and row i - 1 too when i % 3 == 0 (rows shorter in C than
    # in products)
    two = (np.arange(n) % 3 == 0) & (np.arange(n) > 0)
    a_rpt = np.concatenate([[0], np.cumsum(1 + two)]).astype(np.int32)
    a_col = np.repeat(np.arange(n), 1 + two)
    a_col[a_rpt[:-1][two]] -= 1
    A = brm.CSR(n, n, a_rpt, a_col.astype(np.int32), rng.uniform(-1, 1, len(a_col)))
    R = oracle_mod.precise(A, B)
    ctx = brm.Context()
    dA, dB = brm.DeviceCSR.from_host(A), brm.DeviceCSR.from_host(B)
    assert_same_csr(ctx.upper(dA, dB).to_host(), R, "upper")
    assert_same_csr(brm.brmerge_upper(A, B), R, "host upper")
    ctx.close()
