"""Triangular solves whose rows are taken 32 entries at a time by a whole warp:
a dense triangle, so that rows end in every remainder of a chunk, in each
triangle and op; DETERMINISTIC, bit for bit."""

import numpy as np
import pytest

from asc_cpp_b200._abi import (SparseBlasDiagonal, SparseBlasLayout, SparseBlasTranspose,
                               SparseBlasTriangle)
from asc_cpp_b200.sparse_cuda import CudaSparseTriangularSolveMultiple, DenseMatrixView

from gpu_util import bits_equal, context, csr, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("lower", [True, False])
def test_dense_triangle(cuda_lib, restatement, dt, lower):
    n = 199
    rng = np.random.default_rng(n)
    full = rng.uniform(-1, 1, (n, n)) / n
    if np.iscomplexobj(dt(0)):
        full = full + 1j * rng.uniform(-1, 1, (n, n)) / n
    full[np.arange(n), np.arange(n)] += 2
    keep = np.tril(np.ones((n, n), bool)) if lower else np.triu(np.ones((n, n), bool))
    ptr = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int64)
    idx = np.nonzero(keep)[1].astype(np.int64)
    val = full[keep].astype(dt)
    b = (rng.uniform(-1, 1, n) + (1j if np.iscomplexobj(dt(0)) else 0)).astype(dt)
    tri = SparseBlasTriangle.kLower if lower else SparseBlasTriangle.kUpper
    diag = SparseBlasDiagonal.kNonUnit
    ctx = context()
    for op in (SparseBlasTranspose.kNone, SparseBlasTranspose.kTranspose,
               SparseBlasTranspose.kConjugateTranspose):
        x = dev(b)
        CudaSparseTriangularSolveMultiple(ctx, op, 1.25, csr(n, n, ptr, idx, val), tri, diag,
                                          DenseMatrixView(x, n, 1, SparseBlasLayout(1)))
        want = restatement.triangular_solve(int(op), int(tri), int(diag), n, ptr, idx, val, 1.25,
                                            b, 1, None, 1)
        assert bits_equal(host(x), want), op
    ctx.close()
