"""The SpMM row kernel where it can go wrong: rows far longer than the mean
(taken by a warp or a whole block), chunk widths of 16, 8 and 4 bytes, every layout
pair (column-major right-hand sides: the kernel with a lane per row), and a
captured product."""

import numpy as np
import pytest
import torch

from asc_cpp_b200 import synthetic
from asc_cpp_b200._abi import Determinism, SparseBlasLayout, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import CudaSpmm, DenseMatrixView
from oracle import COL_MAJOR, CSR, OP_NONE, ROW_MAJOR

from gpu_util import bits_equal, context, csr, dev, gamma, host

pytestmark = pytest.mark.gpu

ROW, COL = SparseBlasLayout.kRowMajor, SparseBlasLayout.kColumnMajor
ORDER = {ROW: ROW_MAJOR, COL: COL_MAJOR}


def uneven(dt, rows, cols, seed):
    """Short rows, empty rows, and four of 130, 1,000, 5,000 and `cols` entries."""
    rng = np.random.default_rng(seed)
    lengths = rng.integers(0, 24, rows)
    lengths[[3, rows // 2, rows - 2, rows - 1]] = [130, 1000, 5000, cols]
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.permutation(cols)[:n]) for n in lengths]).astype(np.int64)
    return synthetic.Csr(rows, cols, ptr, idx, rng.standard_normal(idx.size).astype(dt)), rng


def operand(rng, rows, k, layout, pad, dt):
    """A stored rows x k operand with `pad` unused elements per row (or column)."""
    ld = (k if layout == ROW else rows) + pad
    return rng.uniform(-1, 1, ld * (rows if layout == ROW else k)).astype(dt), ld


def columns(stored, rows, k, layout, ld):
    return stored.reshape(rows, ld)[:, :k] if layout == ROW else stored.reshape(k, ld)[:, :rows].T


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("k,rows", [(1, 700), (2, 9000), (3, 700), (5, 20_000), (8, 700), (50, 2500),
                                    (130, 700)])
@pytest.mark.parametrize("bl,cl,pad", [(ROW, ROW, 0), (ROW, ROW, 3), (COL, COL, 0), (COL, ROW, 2),
                                       (ROW, COL, 1)])
def test_rows_kernel(cuda_lib, restatement, dt, k, rows, bl, cl, pad):
    cols = 6000
    a_h, rng = uneven(dt, rows, cols, 7 * k + pad)
    b, ldb = operand(rng, cols, k, bl, pad, dt)
    c0, ldc = operand(rng, rows, k, cl, pad, dt)
    a = csr(a_h.rows, a_h.cols, a_h.ptr, a_h.idx, a_h.val)
    for mode in (Determinism.kDeterministic, Determinism.kBackendDefault):
        ctx = context(mode)
        c = dev(c0)
        CudaSpmm(ctx, SparseBlasTranspose.kNone, -1.5, a,
                 DenseMatrixView(dev(b), cols, k, bl, ldb, False),
                 DenseMatrixView(c, rows, k, cl, ldc))
        out = host(c)
        ctx.close()
        if mode == Determinism.kDeterministic:
            expect = c0.copy()
            restatement.standard_spmm(CSR, OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, -1.5, b,
                                      ORDER[bl], ldb, expect, ORDER[cl], ldc, k)
            assert bits_equal(out, expect)
            continue
        # padding keeps its bits; each output within gamma_{n+2} of the exact one
        got = columns(out, rows, k, cl, ldc)
        start = columns(c0, rows, k, cl, ldc)
        kept = out.copy()
        columns(kept, rows, k, cl, ldc)[:] = start
        assert bits_equal(kept, c0)
        counts = restatement.output_counts(OP_NONE, rows, cols, a_h.ptr, a_h.idx)
        for j in {0, k // 2, k - 1}:
            bj = np.ascontiguousarray(columns(b, cols, k, bl, ldb)[:, j])
            exact, absval = restatement.extended(OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, bj)
            ref = start[:, j].astype(np.longdouble) - 1.5 * exact
            bound = gamma(counts + 2, dt) * (1.5 * absval.astype(np.float64) +
                                             np.abs(start[:, j].astype(np.float64)))
            err = np.abs(got[:, j].astype(np.longdouble) - ref).astype(np.float64)
            assert np.all(err <= bound + np.finfo(dt).tiny), j


def test_column_major_under_capture(cuda_lib, restatement):
    """A captured product takes no scratch (a graph would keep its address) and
    gives the same bits."""
    rows, cols, k = 20_000, 6000, 6
    a_h, rng = uneven(np.float64, rows, cols, 5)
    b, c0 = rng.uniform(-1, 1, cols * k), rng.uniform(-1, 1, rows * k)
    a = csr(rows, cols, a_h.ptr, a_h.idx, a_h.val)
    stream = torch.cuda.Stream()
    from asc_cpp_b200.sparse_cuda import SparseCudaContext
    ctx = SparseCudaContext.Create(0, stream=stream)
    bd, c = dev(b), dev(c0)
    args = (ctx, SparseBlasTranspose.kNone, 0.5, a, DenseMatrixView(bd, cols, k, COL, cols, False),
            DenseMatrixView(c, rows, k, COL, rows))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        CudaSpmm(*args)
    graph.replay()
    torch.cuda.synchronize()
    captured = host(c).copy()
    expect = c0.copy()
    restatement.standard_spmm(CSR, OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, 0.5, b, COL_MAJOR,
                              cols, expect, COL_MAJOR, rows, k)
    assert bits_equal(captured, expect)
    c.copy_(dev(c0))
    torch.cuda.synchronize()
    CudaSpmm(*args)
    ctx.synchronize()
    assert bits_equal(host(c), expect)
    del graph
    ctx.close()
