"""The sparse products that a program has this library do, as measurable cases.

A case is a dict of plain values.  ``kind`` names the operation:

* ``spmv``    - ``y = alpha A x + beta y`` (the compat entry point), or, for complex elements,
                ``y += alpha A x`` (the standard entry point, which takes them);
* ``spmv_t``  - ``y += alpha A^T x``;
* ``spmm``    - ``C += alpha A B`` with ``k`` right-hand sides, row- or column-major;
* ``batch``   - one SpMV of each of ``count`` banded matrices, one launch;
* ``trsv``    - a lower triangular solve with one right-hand side;
* ``convert`` - CSR to CSC on the device.

``matrix`` and ``n`` give the operand (``n`` is the number of rows of ``powerlaw`` and ``blocks``,
and the edge of the grid of ``laplacian`` (n x n) and ``stencil`` (n x n x n)), ``mode`` the
numerical mode (``exact``: the bit-exact DETERMINISTIC mode, which a new context has; ``fast``:
BACKEND_DEFAULT), and ``plan`` whether the program keeps a plan of the matrix or calls the plain
entry point.  All matrices are made on the GPU from a seed.
"""

from __future__ import annotations

import math

import torch

from asc_cpp_b200 import sparse_cuda as sc
from asc_cpp_b200._abi import (PLAN_ROW_GROUPS, PLAN_TRANSPOSE, PLAN_TRIANGULAR, Determinism,
                               SparseBlasDiagonal, SparseBlasLayout, SparseBlasTranspose,
                               SparseBlasTriangle)

ALPHA, BETA = 1.5, 0.5
DTYPES = {"f32": torch.float32, "f64": torch.float64,
          "c64": torch.complex64, "c128": torch.complex128}


def listed():
    return [
        # an iteration of an explicit scheme or smoother on a small 2-D grid: the smallest call
        # that programs make over and over, where latency counts
        dict(name="spmv laplacian f64", kind="spmv", matrix="laplacian", n=316, dtype="f64",
             mode="exact", plan=False),
        # graph analytics and Krylov methods on one large irregular matrix, plan kept
        dict(name="spmv powerlaw 4M f64", kind="spmv", matrix="powerlaw", n=4_194_304,
             dtype="f64", mode="fast", plan=True),
        # the same matrix in single precision through the drop-in call, in the mode that a
        # context has when nothing is set
        dict(name="spmv powerlaw 4M f32 exact", kind="spmv", matrix="powerlaw", n=4_194_304,
             dtype="f32", mode="exact", plan=False),
        # frequency-domain operators: complex elements, an odd grid
        dict(name="spmv stencil c128", kind="spmv", matrix="stencil", n=63, dtype="c128",
             mode="exact", plan=False),
        # the adjoint product of a least-squares iteration, drop-in, default mode of a context
        dict(name="spmv_t powerlaw f64", kind="spmv_t", matrix="powerlaw", n=524_287,
             dtype="f64", mode="exact", plan=False),
        # a block of right-hand sides through a 3-D discretisation, plan kept
        dict(name="spmm stencil k32 f32", kind="spmm", matrix="stencil", n=128, k=32,
             dtype="f32", mode="fast", plan=True, layout="row"),
        # block Krylov vectors in column-major storage, a few of them, drop-in
        dict(name="spmm columns k5 f64", kind="spmm", matrix="stencil", n=80, k=5,
             dtype="f64", mode="exact", plan=False, layout="column"),
        # feature aggregation over a graph, a ragged number of features, drop-in
        dict(name="spmm powerlaw k50 f32", kind="spmm", matrix="powerlaw", n=262_144, k=50,
             dtype="f32", mode="fast", plan=False, layout="row"),
        # block-sparse weights times a batch of activations
        dict(name="spmm blocks k128 f32", kind="spmm", matrix="blocks", n=65_536, k=128,
             dtype="f32", mode="fast", plan=True, layout="row"),
        # many uneven banded systems advanced together
        dict(name="batch 512 banded f64", kind="batch", count=512, max_rows=16_384, band=31,
             dtype="f64", mode="fast"),
        # the preconditioner of a solver: a triangle of a grid operator, analysed once
        dict(name="trsv laplacian f64", kind="trsv", matrix="laplacian", n=1000, dtype="f64",
             mode="exact", plan=True),
        # assembly hands over CSR, the next stage wants CSC
        dict(name="convert powerlaw f64", kind="convert", matrix="powerlaw", n=1_048_576,
             dtype="f64"),
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _matrix(rng, most):
    """A matrix of about 10^4 to `most` rows."""
    matrix = rng.choice(["powerlaw", "laplacian", "stencil"])
    rows = _log_int(rng, 10_000, most)
    n = rows if matrix == "powerlaw" else (
        round(rows ** (1 / 2)) if matrix == "laplacian" else round((rows / 2) ** (1 / 3)))
    return dict(matrix=matrix, n=n)


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv_t", "spmm", "spmm", "batch", "trsv", "convert"])
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 64, 512), max_rows=_log_int(rng, 512, 16_384),
                    band=rng.randint(3, 31), dtype=rng.choice(["f64", "f64", "f32"]),
                    mode=rng.choice(["exact", "fast"]))
    if kind == "trsv":
        matrix = rng.choice(["laplacian", "stencil"])
        n = _log_int(rng, 100, 1000) if matrix == "laplacian" else _log_int(rng, 20, 100)
        return dict(kind=kind, matrix=matrix, n=n, dtype=rng.choice(["f64", "f64", "f32"]),
                    mode=rng.choice(["exact", "fast"]), plan=rng.random() < 0.7)
    if kind == "convert":
        return dict(kind=kind, **_matrix(rng, 1_048_576), dtype=rng.choice(["f64", "f32"]))
    if kind == "spmm":
        if rng.random() < 0.2:
            return dict(kind=kind, matrix="blocks", n=16 * _log_int(rng, 256, 4096),
                        k=rng.choice([8, 32, 64, 100, 128]), dtype="f32", mode="fast", plan=True,
                        layout="row")
        k = _log_int(rng, 2, 128)
        layout = rng.choice(["row", "row", "column"])
        most = 16_000_000 if layout == "row" else 5_000_000
        case = dict(kind=kind, **_matrix(rng, most // (k + 20)), k=k,
                    dtype=rng.choice(["f32", "f64"]), mode=rng.choice(["exact", "fast"]),
                    plan=rng.random() < 0.4, layout=layout)
        if case["plan"] and rng.random() < 0.7:
            case["k"] = 4 * -(-k // 4)  # programs that keep a plan mostly pad k
        return case
    if kind == "spmv_t":
        return dict(kind=kind, **_matrix(rng, 524_287), dtype=rng.choice(["f64", "f32"]),
                    mode=rng.choice(["exact", "fast"]), plan=rng.random() < 0.5)
    dtype = rng.choice(["f64", "f64", "f32", "f32", "c128", "c64"])
    return dict(kind=kind, **_matrix(rng, 4_194_304 if dtype[0] == "f" else 300_000), dtype=dtype,
                mode=rng.choice(["exact", "fast"]), plan=rng.random() < 0.5)


# ---- operands ---------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, dtype, gen):
    """Uniform in [-1, 1] (both parts of complex elements)."""
    parts = 2 if dtype.is_complex else 1
    v = torch.rand(n, parts, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    return (torch.view_as_complex(v) if parts == 2 else v[:, 0]).to(dtype).contiguous()


def _normal(n, dtype, gen):
    return torch.randn(n, generator=gen, device="cuda", dtype=dtype)


def _offsets(counts):
    ptr = torch.zeros(counts.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=ptr[1:])
    return ptr


def _structure(matrix, n, gen):
    """(rows, offsets, indices) of a square matrix; indices increase within each row."""
    if matrix == "powerlaw":
        # row lengths lognormal with mean 16 and sigma 1.5, the same for every seed; the L columns
        # of a row are random, one in each of L equal ranges, so distinct and increasing
        mu, longest = math.log(16.0) - 1.5 * 1.5 / 2, min(65_536, n)
        lengths = torch.randn(n, generator=_generator(n), device="cuda", dtype=torch.float64)
        lengths = torch.exp(lengths * 1.5 + mu).round_().clamp_(1, longest).long()
        ptr = _offsets(lengths)
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), lengths)
        j, length = torch.arange(row.numel(), device="cuda") - ptr[row], lengths[row]
        first, end = j * n // length, (j + 1) * n // length
        u = torch.rand(row.numel(), generator=gen, device="cuda", dtype=torch.float64)
        return n, ptr, torch.minimum(first + (u * (end - first)).long(), end - 1)
    if matrix == "blocks":
        # dense 16 x 16 blocks, 2% of the blocks of each block row
        blocks = n // 16
        per = max(1, round(0.02 * blocks))
        pick = torch.rand(blocks, blocks, generator=gen, device="cuda").topk(per, 1).indices
        pick = torch.sort(pick, 1).values * 16
        row = (pick[:, :, None] + torch.arange(16, device="cuda")).reshape(blocks, 1, per * 16)
        idx = row.expand(blocks, 16, per * 16).reshape(-1)
        return n, torch.arange(n + 1, device="cuda") * (per * 16), idx
    if matrix == "laplacian":  # 5 points on an n x n grid
        extents = (n, n)
        steps = [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)]
    else:  # stencil: 27 points on an n^3 grid
        extents = (n, n, n)
        steps = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    rows = n ** len(extents)
    cell = torch.arange(rows, device="cuda")
    at = [(cell // n ** (len(extents) - 1 - d)) % n for d in range(len(extents))]
    valid = torch.empty(rows, len(steps), dtype=torch.bool, device="cuda")
    columns = torch.empty(rows, len(steps), dtype=torch.int64, device="cuda")
    for j, step in enumerate(steps):
        inside = torch.ones(rows, dtype=torch.bool, device="cuda")
        shift = 0
        for d, s in enumerate(step):
            shift = shift * n + s
            if s:
                inside &= (at[d] + s >= 0) & (at[d] + s < n)
        valid[:, j] = inside
        columns[:, j] = cell + shift
    return rows, _offsets(valid.sum(1)), columns[valid]


def _values(case, gen, rows, ptr, idx):
    """Stored values: 4 and -1 for the Laplacian, N(0, 1) otherwise."""
    dtype = DTYPES[case["dtype"]]
    if case["matrix"] == "laplacian":
        row = torch.repeat_interleave(torch.arange(rows, device="cuda"), ptr.diff())
        return torch.where(row == idx, 4.0, -1.0).to(dtype)
    return _normal(idx.numel(), dtype, gen)


def _square(case, gen):
    rows, ptr, idx = _structure(case["matrix"], case["n"], gen)
    return rows, ptr, idx, _values(case, gen, rows, ptr, idx)


def _triangle(case, gen):
    """The lower triangle of a grid operator; a random one gets a dominant diagonal."""
    rows, ptr, idx, val = _square(case, gen)
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), ptr.diff())
    keep = idx <= row
    row, idx, val = row[keep], idx[keep], val[keep]
    if case["matrix"] != "laplacian":
        size = torch.zeros(rows, dtype=val.dtype, device="cuda").index_add_(0, row, val.abs())
        val = torch.where(row == idx, 1 + size[row], val)
    return rows, _offsets(torch.bincount(row, minlength=rows)), idx, val


def _batch(case, seed):
    """`count` banded matrices with 1% entries off the band, back to back; each matrix's entries
    begin at a multiple of 4.  Sizes and half bandwidths are the same for every seed.  (sizes, first
    row, first entry, entries, offsets, indices, values, x, global row of each entry, and where each
    entry is stored)"""
    gen = _generator(seed)
    host = torch.Generator().manual_seed(case["count"])
    count, dtype = case["count"], DTYPES[case["dtype"]]
    sizes = torch.randint(64, case["max_rows"] + 1, (count,), generator=host).cuda()
    bands = torch.randint(1, case["band"] + 1, (count,), generator=host).cuda()
    first = _offsets(sizes)
    total = int(first[-1])
    matrix = torch.repeat_interleave(torch.arange(count, device="cuda"), sizes)
    r = torch.arange(total, device="cuda") - first[matrix]
    lo = (r - bands[matrix]).clamp_(min=0)
    width = torch.minimum(r + bands[matrix], sizes[matrix] - 1) - lo + 1
    start = torch.cumsum(width, 0) - width
    row = torch.repeat_interleave(torch.arange(total, device="cuda"), width)
    keys = (row << 14) | (torch.arange(row.numel(), device="cuda") - start[row] + lo[row])
    extra = torch.randint(0, total, (row.numel() // 100,), generator=gen, device="cuda")
    u = torch.rand(extra.numel(), generator=gen, device="cuda", dtype=torch.float64)
    keys = torch.cat([keys, (extra << 14) | (u * sizes[matrix[extra]]).long()])
    keys = torch.unique_consecutive(torch.sort(keys).values)
    row, col = keys >> 14, keys & ((1 << 14) - 1)
    del keys
    counts = torch.bincount(row, minlength=total)
    ends = _offsets(counts)
    nnz = ends[first[1:]] - ends[first[:-1]]
    base = _offsets((nnz + 3) // 4 * 4)
    place = torch.arange(row.numel(), device="cuda") + (base[:-1] - ends[first[:-1]])[matrix[row]]
    idx = torch.zeros(int(base[-1]), dtype=torch.int64, device="cuda")
    idx[place] = col
    val = _normal(int(base[-1]), dtype, gen)
    x = _uniform(total, dtype, gen)
    # offsets of matrix m: its rows' ends, from 0, with one more entry per matrix
    slot = first[:-1] + torch.arange(count, device="cuda")
    ptr = torch.zeros(total + count, dtype=torch.int64, device="cuda")
    ptr[torch.arange(total, device="cuda") + matrix + 1] = (
        ends[1:] - ends[first[:-1]][matrix])
    return (sizes.tolist(), first.tolist(), base.tolist(), nnz.tolist(), slot.tolist(), ptr, idx,
            val, x, row, place)


# ---- the cases --------------------------------------------------------------

def _context(case):
    fast = case.get("mode") == "fast"
    return sc.SparseCudaContext.Create(
        0, stream=torch.cuda.current_stream(),
        determinism=Determinism.kBackendDefault if fast else Determinism.kDeterministic)


def _dense(case, rows, gen):
    """A rows x k right-hand side in the case's layout, as stored."""
    k = case["k"]
    shape = (rows, k) if case["layout"] == "row" else (k, rows)
    return _normal(rows * k, DTYPES[case["dtype"]], gen).view(shape)


def _view(case, t, rows, writable):
    layout = (SparseBlasLayout.kRowMajor if case["layout"] == "row"
              else SparseBlasLayout.kColumnMajor)
    return sc.DenseMatrixView(t, rows, case["k"], layout, writable=writable)


def prepare(case, seed):
    kind, context = case["kind"], _context(case)
    if kind == "batch":
        sizes, first, base, nnz, slot, ptr, idx, val, x, _, _ = _batch(case, seed)
        y = torch.zeros_like(x)
        matrices, xs, ys = [], [], []
        for m, n in enumerate(sizes):
            b, r = base[m], first[m]
            matrices.append(sc.CudaCsrArray(n, n, ptr[slot[m]:slot[m] + n + 1],
                                            idx[b:b + nnz[m]], val[b:b + nnz[m]]))
            xs.append(sc.CudaStridedVectorView(x, n, 1, r, writable=False))
            ys.append(sc.CudaStridedVectorView(y, n, 1, r))
        work = sc.CudaBatch(context, matrices, xs, ys)
        work.capture(1.0, 0.0)
        return dict(kind=kind, batch=work, y=y)
    gen = _generator(seed)
    if kind == "trsv":
        rows, ptr, idx, val = _triangle(case, gen)
        matrix = sc.CudaCsrArray(rows, rows, ptr, idx, val)
        plan = None
        if case["plan"]:
            plan = sc.CsrPlan(context, matrix, PLAN_TRIANGULAR)
            plan.triangular_analysis(SparseBlasTranspose.kNone, SparseBlasTriangle.kLower)
        b = _uniform(rows, val.dtype, gen)
        x = torch.empty_like(b)
        return dict(kind=kind, context=context, matrix=matrix, plan=plan, b=b, x=x,
                    view=sc.CudaStridedVectorView.of(x))
    rows, ptr, idx, val = _square(case, gen)
    matrix = sc.CudaCsrArray(rows, rows, ptr, idx, val)
    state = dict(kind=kind, context=context, matrix=matrix, plan=None)
    if kind == "convert":
        return state
    if kind == "spmm":
        if case["plan"]:
            state["plan"] = sc.CsrPlan(context, matrix, PLAN_ROW_GROUPS)
        b, c = _dense(case, rows, gen), _dense(case, rows, gen)
        state.update(c=c, bv=_view(case, b, rows, False), cv=_view(case, c, rows, True))
        return state
    x, y = _uniform(rows, val.dtype, gen), _uniform(rows, val.dtype, gen)
    xv, yv = sc.CudaStridedVectorView.of(x, False), sc.CudaStridedVectorView.of(y)
    state.update(y=y, xv=xv, yv=yv, complex=val.dtype.is_complex)
    if case["plan"]:
        state["plan"] = sc.CsrPlan(context, matrix, PLAN_TRANSPOSE if kind == "spmv_t" else 0)
    elif kind == "spmv" and not val.dtype.is_complex:
        need = sc.CudaCsrSpmvWorkspaceSize(context, matrix, xv, yv)
        state["workspace"] = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].spmv(1.0, 0.0)
        return state["y"]
    context, matrix, plan = state["context"], state["matrix"], state["plan"]
    if kind == "convert":
        out = sc.CudaConvertCompressed(context, matrix)
        return out.offsets, out.indices, out.values
    if kind == "trsv":
        state["x"].copy_(state["b"])
        sc.CudaSparseTriangularSolve(context, SparseBlasTranspose.kNone, 1.0, matrix,
                                     SparseBlasTriangle.kLower, SparseBlasDiagonal.kNonUnit,
                                     state["view"], plan)
        return state["x"]
    if kind == "spmm":
        sc.CudaSpmm(context, SparseBlasTranspose.kNone, ALPHA, matrix, state["bv"], state["cv"],
                    plan)
        return state["c"]
    xv, yv = state["xv"], state["yv"]
    if kind == "spmv_t":
        sc.CudaSpmv(context, SparseBlasTranspose.kTranspose, ALPHA, matrix, xv, yv, plan)
    elif state["complex"]:
        sc.CudaSpmv(context, SparseBlasTranspose.kNone, ALPHA, matrix, xv, yv, plan)
    elif plan is not None:
        plan.csr_spmv(ALPHA, xv, BETA, yv)
    else:
        sc.CudaCsrSpmv(context, ALPHA, matrix, xv, BETA, yv, state["workspace"])
    return state["y"]


def _size(case):
    """(rows, expected stored entries) of the case's matrix."""
    matrix, n = case["matrix"], case["n"]
    if matrix == "powerlaw":
        return n, 16 * n
    if matrix == "blocks":
        return n, n * 16 * max(1, round(0.02 * (n // 16)))
    if matrix == "laplacian":
        return n * n, 5 * n * n - 4 * n
    return n ** 3, (3 * n - 2) ** 3


def work(case):
    """Stored entries once (value and 8-byte index), offsets, inputs and outputs once."""
    element = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}[case["dtype"]]
    kind, terms = case["kind"], 8 if case["dtype"][0] == "c" else 2
    if kind == "batch":
        rows = case["count"] * (64 + case["max_rows"]) / 2
        nnz = rows * (case["band"] + 2) * 1.01
        return dict(bytes=nnz * (8 + element) + rows * (8 + 2 * element), flops=2 * nnz)
    rows, nnz = _size(case)
    if kind == "convert":
        return dict(bytes=2 * (nnz * (8 + element) + 8 * (rows + 1)), flops=0)
    if kind == "trsv":
        nnz = (nnz + rows) // 2
        return dict(bytes=nnz * (8 + element) + 8 * (rows + 1) + 2 * rows * element, flops=2 * nnz)
    k = case.get("k", 1)
    return dict(bytes=nnz * (8 + element) + 8 * (rows + 1) + 3 * rows * k * element,
                flops=terms * nnz * k)


def _product(ptr, idx, val, x):
    """A x (or A X) in 64 bits, real or complex."""
    if val.dtype.is_complex:
        parts = [_product(ptr, idx, v, torch.view_as_real(x.to(torch.complex128)))
                 for v in (val.real, val.imag)]
        re = parts[0][:, 0] - parts[1][:, 1]
        return torch.complex(re, parts[0][:, 1] + parts[1][:, 0])
    n = ptr.numel() - 1
    a = torch.sparse_csr_tensor(ptr, idx, val.double(), size=(n, n))
    return a @ x.double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        _, first, _, _, _, _, idx, val, x, row, place = _batch(case, seed)
        begin = torch.tensor(first[:-1], device="cuda")
        sizes = torch.tensor(first[1:], device="cuda") - begin
        matrix = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
        columns = idx[place] + begin[matrix[row]]
        terms = val[place].double() * x.double()[columns]
        return torch.zeros(x.numel(), dtype=torch.float64, device="cuda").index_add_(0, row, terms)
    gen = _generator(seed)
    if kind == "trsv":
        rows, ptr, idx, val = _triangle(case, gen)
        b = _uniform(rows, val.dtype, gen)
        a = torch.sparse_csr_tensor(ptr, idx, val.double(), size=(rows, rows))
        return torch.triangular_solve(b.double()[:, None], a, upper=False).solution[:, 0]
    rows, ptr, idx, val = _square(case, gen)
    if kind == "convert":
        order = torch.sort(idx, stable=True).indices
        row = torch.repeat_interleave(torch.arange(rows, device="cuda"), ptr.diff())
        return (_offsets(torch.bincount(idx, minlength=rows)), row[order], val[order].double())
    if kind == "spmm":
        b, c = _dense(case, rows, gen), _dense(case, rows, gen)
        if case["layout"] == "row":
            return c.double() + ALPHA * _product(ptr, idx, val, b)
        return c.double() + ALPHA * _product(ptr, idx, val, b.t().contiguous()).t()
    x, y = _uniform(rows, val.dtype, gen), _uniform(rows, val.dtype, gen)
    wide = torch.complex128 if val.dtype.is_complex else torch.float64
    if kind == "spmv_t":
        row = torch.repeat_interleave(torch.arange(rows, device="cuda"), ptr.diff())
        return y.to(wide).index_add_(0, idx, ALPHA * val.to(wide) * x.to(wide)[row])
    beta = 1.0 if val.dtype.is_complex else BETA
    return beta * y.to(wide) + ALPHA * _product(ptr, idx, val, x)
