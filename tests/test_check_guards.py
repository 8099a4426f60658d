"""Every store of the rank, pack and segment kernels to a shared-memory slot (or
the long-column scratch) whose index is a computed rank has its bounds check of
the checked build (brm_check.cuh) in front of it."""
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "brmerge_gb300" / "csrc"

STORES = [
    ("brm_midrank.cuh", "atomicOr(&cw[ci], b);", 1), ("brm_midrank.cuh", "ucol[r] = c[u];", 1),
    ("brm_midrank.cuh", "mlist[o + __popc(mb & ltm)] =", 1),
    ("brm_midrank.cuh", "quads[o++] =", 2), ("brm_midrank.cuh", "vals[p] = vmul(", 1),
    ("brm_rankpack.cuh", "atomicOr(&cw[ci], b);", 1), ("brm_rankpack.cuh", "ucol[r] = c[u];", 1),
    ("brm_rankpack.cuh", "mlist[nm + __popc(mb & ltm)] =", 1),
    ("brm_rankpack.cuh", "quads[o++] =", 1), ("brm_rankpack.cuh", "vals[p] = vmul(", 1),
    ("brm_seg.cuh", "atomicOr(&cw[ci], b);", 1), ("brm_seg.cuh", "ucol[r] = c[u];", 1),
    ("brm_seg.cuh", "lista[o] =", 1), ("brm_seg.cuh", "vals[p] = vmul(", 1),
    ("brm_seg.cuh", "P.long_leaf[leo + r] =", 1)]


@pytest.mark.parametrize("name,store,times", STORES)
def test_store_is_guarded(name, store, times):
    lines = (CSRC / name).read_text().splitlines()
    at = [i for i, line in enumerate(lines) if store in line]
    assert len(at) == times
    for i in at:
        assert any("BRM_IN(P.cnt" in line for line in lines[i - 3:i]), f"{name}:{i + 1}"
