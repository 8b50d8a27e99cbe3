"""SpMM with few long rows (four lanes a row whatever the width): both sides of the
rule's edges in rows and in mean length, and rows that are set aside."""

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


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 6, 8, 12])
@pytest.mark.parametrize("case", ["one", "few", "short", "fast edge", "edge", "past"])
def test_few_rows(cuda_lib, restatement, dt, k, case):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = {"one": 1, "few": 1003, "short": 1003, "fast edge": sms * 256,
            "edge": sms * 320, "past": sms * 320 + 1}[case]
    if rows > 2000 and k not in (1, 3, 8):
        pytest.skip("the edge in rows at three widths")
    cols = 3000
    rng = np.random.default_rng(k)
    lengths = np.full(rows, 32, np.int64)
    if case == "one":
        lengths[0] = 2999
    elif case == "few":
        lengths[[5, 700]] = [0, 1500]  # set aside
    elif case == "short":
        lengths[17] = 31  # one entry short of the mean
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    first = rng.integers(0, cols - lengths + 1)
    idx = np.repeat(first - ptr[:-1], lengths) + np.arange(ptr[-1])
    val = rng.standard_normal(idx.size, dtype=dt)
    a_h = synthetic.Csr(rows, cols, ptr, idx.astype(np.int64), val)
    b = rng.standard_normal(cols * k, dtype=dt)
    c0 = rng.standard_normal(rows * k, dtype=dt)
    a = csr(rows, cols, a_h.ptr, a_h.idx, a_h.val)
    for mode in (Determinism.kDeterministic, Determinism.kBackendDefault):
        ctx = context(mode)
        c = dev(c0)
        CudaSpmm(ctx, SparseBlasTranspose.kNone, 0.75, a, DenseMatrixView(dev(b), cols, k, ROW, k, False),
                 DenseMatrixView(c, rows, k, ROW, k))
        got = host(c)
        ctx.close()
        if mode == Determinism.kDeterministic:
            expect = c0.copy()
            restatement.standard_spmm(CSR, OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, 0.75, b,
                                      ROW_MAJOR, k, expect, ROW_MAJOR, k, k)
            assert bits_equal(got, expect)
            continue
        counts = restatement.output_counts(OP_NONE, rows, cols, a_h.ptr, a_h.idx)
        for j in {0, k - 1}:
            bj = np.ascontiguousarray(b.reshape(cols, k)[:, j])
            exact, absval = restatement.extended(OP_NONE, rows, cols, a_h.ptr, a_h.idx, a_h.val, bj)
            start = c0.reshape(rows, k)[:, j]
            ref = start.astype(np.longdouble) + 0.75 * exact
            bound = gamma(counts + 2, dt) * (0.75 * absval.astype(np.float64) +
                                             np.abs(start.astype(np.float64)))
            err = np.abs(got.reshape(rows, k)[:, j].astype(np.longdouble) - ref).astype(np.float64)
            assert np.all(err <= bound + np.finfo(dt).tiny), j
