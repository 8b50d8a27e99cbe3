"""SpMM where a block meets more long rows than it can set aside at a time: the
contracted form adds every row up the same way on every run, and the
deterministic form keeps its bits."""

import numpy as np
import pytest
import torch

from asc_cpp_b200 import synthetic
from asc_cpp_b200._abi import Determinism, SparseBlasLayout, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import CudaSpmm, DenseMatrixView
from oracle import CSR, OP_NONE, ROW_MAJOR

from gpu_util import bits_equal, context, csr, dev, gamma, host

pytestmark = pytest.mark.gpu

ROW = SparseBlasLayout.kRowMajor


def many_long(dt, rows, cols, every, length, seed):
    """One entry a row; each `every`-th row has `length` to `length` + 15."""
    rng = np.random.default_rng(seed)
    lengths = np.ones(rows, np.int64)
    lengths[::every] = length + rng.integers(0, 16, lengths[::every].size)
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    first = rng.integers(0, cols - 2 * lengths + 2)
    idx = np.repeat(first - 2 * ptr[:-1], lengths) + 2 * np.arange(ptr[-1])
    val = rng.standard_normal(idx.size, dtype=dt)
    return synthetic.Csr(rows, cols, ptr, idx.astype(np.int64), val), rng


# `per_block`: rows of the blocks of the grid, 4 or 8 to an SM.  The last
# matrix has too many rows beyond four times the limit as well.
@pytest.mark.parametrize("dt,k,per_sm,per_block,every,length", [
    (np.float32, 16, 4, 1000, 12, 130),
    (np.float64, 8, 4, 1000, 12, 130),
    (np.float32, 4, 8, 1000, 12, 130),
    (np.float64, 3, 8, 1000, 12, 130),
    (np.float32, 50, 8, 1000, 12, 130),
    (np.float32, 16, 4, 3600, 50, 600)])
def test_many_long_rows(cuda_lib, restatement, dt, k, per_sm, per_block, every, length):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, cols = sms * per_sm * per_block + 5, 4096
    a_h, rng = many_long(dt, rows, cols, every, length, k)
    b = rng.standard_normal(cols * k, dtype=dt)
    c0 = rng.standard_normal(rows * k, dtype=dt)
    a = csr(rows, cols, a_h.ptr, a_h.idx, a_h.val)
    bv = DenseMatrixView(dev(b), cols, k, ROW, k, False)

    def product(mode):
        ctx = context(mode)
        c = dev(c0)
        CudaSpmm(ctx, SparseBlasTranspose.kNone, -1.5, a, bv, DenseMatrixView(c, rows, k, ROW, k))
        out = host(c)
        ctx.close()
        return out

    expect = c0.copy()
    restatement.standard_spmm(CSR, OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, -1.5, b,
                              ROW_MAJOR, k, expect, ROW_MAJOR, k, k)
    assert bits_equal(product(Determinism.kDeterministic), expect)

    first = product(Determinism.kBackendDefault)
    for _ in range(5):
        assert bits_equal(product(Determinism.kBackendDefault), first)
    counts = restatement.output_counts(OP_NONE, rows, cols, a_h.ptr, a_h.idx)
    bj = np.ascontiguousarray(b.reshape(cols, k)[:, 0])
    exact, absval = restatement.extended(OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, bj)
    start = c0.reshape(rows, k)[:, 0]
    ref = start.astype(np.longdouble) - 1.5 * exact
    bound = gamma(counts + 2, dt) * (1.5 * absval.astype(np.float64) +
                                     np.abs(start.astype(np.float64)))
    err = np.abs(first.reshape(rows, k)[:, 0].astype(np.longdouble) - ref).astype(np.float64)
    assert np.all(err <= bound + np.finfo(dt).tiny)
