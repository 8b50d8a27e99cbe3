"""SpMM with more than 32 chunks of 16 bytes per row of B: a warp per row where
rows average 12 or more entries, half a warp in passes where they are shorter;
DETERMINISTIC, bit for bit."""

import numpy as np
import pytest

from asc_cpp_b200._abi import Determinism, SparseBlasLayout, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import CudaSpmm, DenseMatrixView
from oracle import COL_MAJOR, CSR, OP_NONE, ROW_MAJOR

from gpu_util import bits_equal, context, csr, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,k", [(np.float32, 128), (np.float32, 132), (np.float32, 260),
                                  (np.float64, 66), (np.float64, 130)])
@pytest.mark.parametrize("most", [3, 30])
@pytest.mark.parametrize("layout", [SparseBlasLayout.kRowMajor, SparseBlasLayout.kColumnMajor])
def test_wide_rows(cuda_lib, restatement, dt, k, most, layout):
    rows, cols = 1201, 900
    rng = np.random.default_rng(k + most)
    lengths = rng.integers(0, most + 1, rows)
    lengths[[5, rows - 1]] = [129, 700]  # by the whole block
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.permutation(cols)[:n]) for n in lengths]).astype(np.int64)
    val = rng.standard_normal(idx.size).astype(dt)
    b = rng.uniform(-1, 1, cols * k).astype(dt)
    c0 = rng.uniform(-1, 1, rows * k).astype(dt)
    row_major = layout == SparseBlasLayout.kRowMajor
    ldc = k if row_major else rows
    ctx = context(Determinism.kDeterministic)
    c = dev(c0)
    CudaSpmm(ctx, SparseBlasTranspose.kNone, -1.5, csr(rows, cols, ptr, idx, val),
             DenseMatrixView(dev(b), cols, k, SparseBlasLayout.kRowMajor, k, False),
             DenseMatrixView(c, rows, k, layout, ldc))
    out = host(c)
    ctx.close()
    expect = c0.copy()
    restatement.standard_spmm(CSR, OP_NONE, rows, cols, ptr, idx, val, -1.5, b, ROW_MAJOR, k,
                              expect, ROW_MAJOR if row_major else COL_MAJOR, ldc, k)
    assert bits_equal(out, expect)
