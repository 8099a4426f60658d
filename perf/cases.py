"""The products that are timed: what programs have this library do, from a call
of a few hundred rows to a 27-point stencil on 128^3 points.

A case names a call (`form`), a matrix family and its sizes, and a value type:

* precise, upper -- the one-call device forms;
* split          -- the symbolic phase, C allocated by the caller, the numeric phase;
* numeric        -- the numeric phase on a plan that is kept (new values, same structure);
* batch, pipe    -- many independent pairs in one call, allocated by the call or run
                    through a pipeline captured for their capacities;
* host           -- the drop-in on host arrays;
* mtx            -- a MatrixMarket file read into device CSR.

Inputs are made on the GPU.  A case has one structure, which the seed turns:
rows and columns are renumbered cyclically (not the stencil's), so the products
and entries of C are as many for every seed.  Columns are sorted and distinct
within a row, values, from the seed, U[-1, 1) (the stencil: 26 and -1 with a
little jitter).
"""
import functools
import json
import math
import tempfile
import zlib
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

import brmerge_gb300 as brm

DEV = "cuda"


# ---------------------------------------------------------------------------
# Matrices on the GPU
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(n, g):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1


def _pointers(lens):
    rpt = torch.zeros(lens.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=rpt[1:])
    return rpt


def _random_columns(lens, ncols, g):
    """Sorted distinct columns for rows of the given lengths; ncols: the
    number of columns, one for all rows or one a row.  Sorted draws with
    repetition from [0, ncols - len] plus their rank in the row are distinct."""
    rpt = _pointers(lens)
    nnz = int(rpt[-1])
    row = torch.repeat_interleave(torch.arange(lens.numel(), device=DEV), lens, output_size=nnz)
    room = (ncols - lens + 1)[row]
    x = (torch.rand(nnz, generator=g, device=DEV, dtype=torch.float64) * room).to(torch.int64)
    key = torch.sort((row << 32) | torch.minimum(x, room - 1)).values
    return rpt, (key & 0xFFFFFFFF) + torch.arange(nnz, device=DEV) - rpt[row]


def _lognormal_lengths(rows, ncols, cap, g, mu=math.log(6.0), sigma=0.8):
    z = torch.randn(rows, generator=g, device=DEV, dtype=torch.float64)
    lens = torch.floor(torch.exp(mu + sigma * z) + 0.5).to(torch.int64)
    return torch.minimum(lens, torch.as_tensor(ncols, device=DEV)).clamp(max=cap)


def _lengths_family(kind, rows, ncols, per_row, g):
    if kind == "er":  # the same number of entries in every row
        return torch.full((rows,), min(per_row, ncols), dtype=torch.int64, device=DEV)
    if kind == "uniform":  # 0 .. per_row entries, empty rows among them
        return torch.randint(0, min(per_row, ncols) + 1, (rows,), generator=g, device=DEV)
    return _lognormal_lengths(rows, ncols, min(per_row, ncols), g)


def _rmat(n, edges, g):
    """R-MAT (.57, .19, .19, .05): `edges` samples on the next power of two,
    scaled to n x n, duplicates removed."""
    bits = max(1, (n - 1).bit_length())
    r = torch.zeros(edges, dtype=torch.int64, device=DEV)
    c = torch.zeros(edges, dtype=torch.int64, device=DEV)
    for _ in range(bits):
        u = torch.rand(edges, generator=g, device=DEV, dtype=torch.float64)
        r = (r << 1) | (u >= 0.76)
        c = (c << 1) | (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    key = torch.unique((((r * n) >> bits) << 32) | ((c * n) >> bits))
    lens = torch.bincount(key >> 32, minlength=n)
    return _pointers(lens), key & 0xFFFFFFFF


def _stencil27(nx, ny, nz):
    n = nx * ny * nz
    idx = torch.arange(n, device=DEV)
    x, y, z = idx % nx, (idx // nx) % ny, idx // (nx * ny)
    cols, oks = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                oks.append((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny)
                           & (z + dz >= 0) & (z + dz < nz))
                cols.append((idx + (dz * ny + dy) * nx + dx).to(torch.int32))
    ok = torch.stack(oks, 1)
    return _pointers(ok.sum(1)), torch.stack(cols, 1)[ok].to(torch.int64)


def _matrix(M, N, rpt, col, val):
    return SimpleNamespace(M=M, N=N, rpt=rpt, col=col, val=val)


def _structure_gen(case):
    """The generator of the case's structure, whatever the seed."""
    sizes = {k: v for k, v in case.items() if k not in ("name", "form", "dtype", "validate")}
    return _gen(zlib.crc32(json.dumps(sizes, sort_keys=True).encode()))


def _turned(M, N, rpt, col, row_shift, col_shift):
    """The structure with its rows and columns renumbered cyclically."""
    row = torch.repeat_interleave(torch.arange(M, device=DEV), rpt.diff())
    key = torch.sort((((row + row_shift) % M) << 32) | ((col + col_shift) % N)).values
    return _pointers(torch.bincount(key >> 32, minlength=M)), key & 0xFFFFFFFF


def _operands(case, seed):
    """(A, B) in 64 bits (indices and values); B is A where the case squares."""
    gs, g = _structure_gen(case), _gen(seed)
    shift = torch.randint(0, 1 << 30, (3,), generator=g, device=DEV).tolist()
    kind = case["matrix"]
    if kind == "rmat":
        n = case["n"]
        rpt, col = _rmat(n, int(case["edge_factor"] * n), gs)
        rpt, col = _turned(n, n, rpt, col, shift[0], shift[0])
        A = _matrix(n, n, rpt, col, _uniform(col.numel(), g))
    elif kind == "stencil27":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        rpt, col = _stencil27(nx, ny, nz)
        row = torch.repeat_interleave(torch.arange(n, device=DEV), rpt.diff())
        val = torch.where(col == row, 26.0, -1.0).to(torch.float64)
        A = _matrix(n, n, rpt, col, val + 1e-3 * _uniform(col.numel(), g))
    else:
        M, K, N, p = case["M"], case["K"], case["N"], case["per_row"]
        square = case["square"]
        rpt, col = _random_columns(_lengths_family(kind, M, K, p, gs), K, gs)
        rpt, col = _turned(M, K, rpt, col, shift[1 if square else 0], shift[1])
        A = _matrix(M, K, rpt, col, _uniform(col.numel(), g))
        if not square:
            rpt, col = _random_columns(_lengths_family(kind, K, N, p, gs), N, gs)
            rpt, col = _turned(K, N, rpt, col, shift[1], shift[2])
            return A, _matrix(K, N, rpt, col, _uniform(col.numel(), g))
    return A, A


def _stack(n, gs, g, col_shift):
    """Square matrices of n[i] rows, lognormal rows, stacked: row pointers
    over all of them, each one's own columns, renumbered by col_shift."""
    width = torch.repeat_interleave(n, n)  # columns of each row's matrix
    rpt, col = _random_columns(_lognormal_lengths(width.numel(), width, 256, gs), width, gs)
    if col_shift:
        row = torch.repeat_interleave(torch.arange(width.numel(), device=DEV), rpt.diff())
        col = torch.sort((row << 32) | ((col + col_shift) % width[row])).values & 0xFFFFFFFF
    return SimpleNamespace(rpt=rpt, col=col, val=_uniform(col.numel(), g))


def _batch_operands(case, seed):
    """(rows of each pair, the A_i stacked, the B_i stacked)."""
    gs, g = _structure_gen(case), _gen(seed)
    n = torch.randint(case["n_min"], case["n_max"] + 1, (case["pairs"],), generator=gs, device=DEV)
    shift = int(torch.randint(1, 1 << 30, (1,), generator=g, device=DEV))
    return n.tolist(), _stack(n, gs, g, 0), _stack(n, gs, g, shift)


def _torch_type(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _device_csr(X, dtype):
    return brm.DeviceCSR(X.M, X.N, X.rpt.to(torch.int32), X.col.to(torch.int32), X.val.to(dtype))


def _host_csr(X, dtype):
    return brm.CSR(X.M, X.N, X.rpt.to(torch.int32).cpu().numpy(),
                   X.col.to(torch.int32).cpu().numpy(), X.val.to(dtype).cpu().numpy())


def _split_stack(S, ns, dtype):
    """The stacked matrices as DeviceCSR of their own, views of three arrays."""
    nm = len(ns)
    n = torch.tensor(ns, dtype=torch.int64, device=DEV)
    first = torch.zeros(nm + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(n, 0, out=first[1:])
    mat = torch.repeat_interleave(torch.arange(nm, device=DEV), n + 1)
    at = torch.arange(mat.numel(), device=DEV) - mat
    start = S.rpt[first]
    rpt = (S.rpt[at] - start[mat]).to(torch.int32)
    rpts = torch.split(rpt, [m + 1 for m in ns])
    sizes = start.diff().tolist()
    cols = torch.split(S.col.to(torch.int32), sizes)
    vals = torch.split(S.val.to(dtype), sizes)
    return [brm.DeviceCSR(ns[i], ns[i], rpts[i], cols[i], vals[i]) for i in range(nm)]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _case(name, form, dtype, matrix, validate=False, **sizes):
    c = {"name": name, "form": form, "dtype": dtype, "matrix": matrix, "validate": validate}
    return {**c, **sizes}


def listed():
    return [
        # one of the many small products of a coarse level or a small graph:
        # launches and synchronisations are all there is
        _case("uniform_300", "precise", "f64", "uniform", M=300, K=250, N=350, per_row=12,
              square=False),
        # the reference's CPU workload: short rows of equal length
        _case("er_16384", "precise", "f64", "er", M=16384, K=16384, N=16384, per_row=8,
              square=True),
        # a served graph query: the denser power-law graph in single precision
        _case("rmat_65536_f32", "precise", "f32", "rmat", n=65536, edge_factor=8.0),
        # the power-law workload: hub rows of up to a million products beside
        # rows of one or two
        _case("rmat_262144", "precise", "f64", "rmat", n=262144, edge_factor=2.35),
        # the same through the upper-bound method
        _case("rmat_262144_upper", "upper", "f64", "rmat", n=262144, edge_factor=2.35),
        # a Galerkin-like product of a large regular grid: the largest call
        _case("stencil_128", "precise", "f64", "stencil27", nx=128, ny=128, nz=128),
        # new values on a kept plan, every step of an iteration (odd sizes)
        _case("stencil_61x47x53_numeric", "numeric", "f64", "stencil27", nx=61, ny=47, nz=53),
        # interpolation-like rectangular operands, symbolic and numeric called
        # apart, inputs checked
        _case("lognormal_rect_split", "split", "f64", "lognormal", validate=True, M=60001, K=50021,
              N=70001, per_row=256, square=False),
        # thousands of uneven pairs in one call
        _case("batch_4096", "batch", "f64", "lognormal", pairs=4096, n_min=256, n_max=8192),
        # a stream of smaller batches through a captured pipeline
        _case("pipe_700_f32", "pipe", "f32", "lognormal", pairs=700, n_min=100, n_max=3000),
        # a host program that swaps the reference's call for this one
        _case("host_rmat_131072", "host", "f64", "rmat", n=131072, edge_factor=2.35),
        # loading the matrix of such a program
        _case("mtx_rmat_100003", "mtx", "f64", "rmat", n=100003, edge_factor=3.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["precise", "precise", "precise", "upper", "upper", "split", "numeric",
                       "numeric", "batch", "pipe", "host", "mtx"])
    dtype = rng.choice(["f64", "f64", "f32"])
    head = {"form": form, "dtype": dtype, "validate": form != "numeric" and rng.random() < 0.2}
    if form in ("batch", "pipe"):
        lo = _log(rng, 32, 2048)
        hi = _log(rng, lo, 8192)
        # about 80 products a row
        return {**head, "matrix": "lognormal", "validate": False, "n_min": lo, "n_max": hi,
                "pairs": _log(rng, 4, max(5, min(2000, 8_000_000 // (lo + hi))))}
    kind = rng.choice(["rmat", "rmat", "stencil27", "stencil27", "er", "uniform", "lognormal"])
    if form == "mtx":
        n = _log(rng, 200, 200_000)
        return {**head, "matrix": "rmat", "n": n, "edge_factor": round(rng.uniform(1.0, 3.0), 3)}
    if kind == "rmat":
        n = _log(rng, 500, 262_144)
        return {**head, "matrix": kind, "n": n,
                "edge_factor": round(rng.uniform(1.0, 8.0 if n <= 65_536 else 2.4), 3)}
    if kind == "stencil27":
        most = 128 if form in ("precise", "upper") else 80
        return {**head, "matrix": kind, "nx": _log(rng, 3, most), "ny": _log(rng, 3, most),
                "nz": _log(rng, 3, most)}
    M, K, N = (_log(rng, 100, 200_000) for _ in range(3))
    if square := rng.random() < 0.4:
        K = N = M
    per_row = {"er": _log(rng, 2, 40), "uniform": _log(rng, 2, 60), "lognormal": 256}[kind]
    return {**head, "matrix": kind, "M": M, "K": K, "N": N, "per_row": per_row, "square": square}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    form, dtype = case["form"], _torch_type(case)
    s = SimpleNamespace(form=form)
    if form == "host":
        A, B = _operands(case, seed)
        s.A = _host_csr(A, dtype)
        s.B = s.A if B is A else _host_csr(B, dtype)
        return s
    s.ctx = brm.Context(validate=case["validate"])
    if form in ("batch", "pipe"):
        ns, SA, SB = _batch_operands(case, seed)
        s.pairs = list(zip(_split_stack(SA, ns, dtype), _split_stack(SB, ns, dtype)))
        if form == "pipe":
            s.pipe = s.ctx.batch_pipe(s.pairs)
        return s
    A, B = _operands(case, seed)
    if form == "mtx":
        s.np_dtype = np.float64 if case["dtype"] == "f64" else np.float32
        s.dir = tempfile.TemporaryDirectory()
        s.path = Path(s.dir.name) / "a.mtx"
        rows = torch.repeat_interleave(torch.arange(1, A.M + 1, device=DEV), A.rpt.diff())
        body = "\n".join(f"{r} {c} {v!r}" for r, c, v in zip(
            rows.tolist(), (A.col + 1).tolist(), A.val.tolist()))
        s.path.write_text("%%MatrixMarket matrix coordinate real general\n"
                          f"{A.M} {A.N} {A.col.numel()}\n{body}\n")
        return s
    s.A = _device_csr(A, dtype)
    s.B = s.A if B is A else _device_csr(B, dtype)
    if form == "numeric":
        s.crpt, s.cnnz = s.ctx.symbolic(s.A, s.B)
        s.out = (torch.empty(s.cnnz, dtype=torch.int32, device=DEV),
                 torch.empty(s.cnnz, dtype=dtype, device=DEV))
    return s


class _Views(dict):
    """Outputs that are views of a pipeline's own arrays; they keep it alive."""

    def __init__(self, owner, **outputs):
        super().__init__(outputs)
        self.owner = owner


def run(s):
    if s.form in ("precise", "upper"):
        C = (s.ctx.precise_device if s.form == "precise" else s.ctx.upper)(s.A, s.B)
    elif s.form == "split":
        crpt, cnnz = s.ctx.symbolic(s.A, s.B)
        C = s.ctx.numeric(s.A, s.B, crpt, cnnz)
    elif s.form == "numeric":
        C = s.ctx.numeric(s.A, s.B, s.crpt, s.cnnz, out=s.out)
    elif s.form == "host":
        C = brm.brmerge_precise(s.A, s.B)
    elif s.form == "mtx":
        C = s.ctx.read_mtx_device(s.path, dtype=s.np_dtype)
    elif s.form == "batch":
        crpt, ccol, cval, row_off, nnz_off, rpt_local = s.ctx.batch_precise_raw(s.pairs)
        return {"rpt": crpt, "col": ccol, "val": cval, "row_off": row_off, "nnz_off": nnz_off,
                "rpt_local": rpt_local}
    else:
        ccol, cval, row_off, nnz_off, rpt_local, nnz = s.pipe.run_raw(s.pairs)
        return _Views(s.pipe, col=ccol, val=cval, row_off=row_off, nnz_off=nnz_off,
                      rpt_local=rpt_local, nnz=nnz)
    return {"rpt": C.rpt, "col": C.col, "val": C.val}


# ---------------------------------------------------------------------------
# What a pass needs, and what it returns in 64 bits
# ---------------------------------------------------------------------------
def _products_in_64_bits(A, B, ncols, values=True):
    """(products, nnz(C), values of C in row and column order) of CSR
    operands with 64-bit arrays, by sorting the products of blocks of rows."""
    lens = B.rpt.diff()[A.col]
    pre = _pointers(lens)
    row_pre = pre[A.rpt]
    total, M = int(pre[-1]), A.rpt.numel() - 1
    nnz, out, r0 = 0, [], 0
    while r0 < M:
        lim = int(row_pre[r0]) + 150_000_000
        r1 = min(M, max(r0 + 1, int(torch.searchsorted(row_pre, lim, right=True)) - 1))
        a0, a1 = int(A.rpt[r0]), int(A.rpt[r1])
        n = int(row_pre[r1] - row_pre[r0])
        if n:
            e = torch.repeat_interleave(torch.arange(a0, a1, device=DEV), lens[a0:a1],
                                        output_size=n)
            at = B.rpt[A.col[e]] + torch.arange(n, device=DEV) + pre[a0] - pre[e]
            row = torch.searchsorted(A.rpt, e, right=True) - 1
            key, order = torch.sort(row * ncols + B.col[at])
            first = torch.ones(n, dtype=torch.bool, device=DEV)
            first[1:] = key[1:] != key[:-1]
            slot = torch.cumsum(first, 0) - 1
            k = int(slot[-1]) + 1
            nnz += k
            if values:
                v = (A.val[e] * B.val[at])[order]
                out.append(torch.zeros(k, dtype=torch.float64, device=DEV).index_add_(0, slot, v))
        r0 = r1
    return total, nnz, torch.cat(out) if out else torch.zeros(0, dtype=torch.float64, device=DEV)


def _rounded(X, dtype):
    """X with its values as the call gets them, in 64 bits again."""
    return SimpleNamespace(rpt=X.rpt, col=X.col, val=X.val.to(dtype).to(torch.float64))


def _stacked_operands(case, seed):
    ns, A, B = _batch_operands(case, seed)
    n = torch.tensor(ns, dtype=torch.int64, device=DEV)
    first = torch.repeat_interleave(torch.cumsum(n, 0) - n, n)  # of each row's matrix
    A.col = A.col + torch.repeat_interleave(first, A.rpt.diff())
    return A, B, max(ns)


def exact(case, seed):
    dtype = _torch_type(case)
    if case["form"] in ("batch", "pipe"):
        A, B, ncols = _stacked_operands(case, seed)
        return {"val": _products_in_64_bits(_rounded(A, dtype), _rounded(B, dtype), ncols)[2]}
    A, B = _operands(case, seed)
    if case["form"] == "mtx":
        return {"val": A.val}
    A, B, ncols = _rounded(A, dtype), _rounded(B, dtype), B.N
    val = _products_in_64_bits(A, B, ncols)[2]
    return {"rpt": None, "col": None, "val": val}


@functools.lru_cache(maxsize=64)
def _counts(items):
    """(entries and rows of A, of B (0 where B is A), rows and entries of C,
    products) of the case, of one seed's inputs: seeds differ little."""
    case = dict(items)
    if case["form"] in ("batch", "pipe"):
        A, B, ncols = _stacked_operands(case, 1)
        same = False
    else:
        A, B = _operands(case, 1)
        ncols, same = B.N, B is A
    na, ra = A.col.numel(), A.rpt.numel()
    nb, rb = (0, 0) if same else (B.col.numel(), B.rpt.numel())
    if case["form"] == "mtx":
        return na, ra, 0, 0, 0, 0, 0
    products, nnz, _ = _products_in_64_bits(A, B, ncols, values=False)
    return na, ra, nb, rb, ra, nnz, products


def work(case):
    na, ra, nb, rb, rc, nc, products = _counts(tuple(sorted(
        (k, v) for k, v in case.items() if k != "name")))
    v = 8 if case["dtype"] == "f64" else 4
    if case["form"] == "mtx":
        # the text (about 31 bytes an entry at these sizes) in, CSR out
        return {"bytes": 31 * na + 4 * ra + (4 + v) * na, "flops": 0}
    return {"bytes": 4 * (ra + rb + rc) + (4 + v) * (na + nb + nc), "flops": 2 * products}
