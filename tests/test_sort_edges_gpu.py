"""The radix sort behind conversions and transposed structures at the edges of
its tiles (4096 entries), digits (1 to 8 bits, 1 to 4 passes), element sizes
and word widths (inner indices past 32 bits take 64-bit words).  Integer work
and moved values: identical to a stable sort."""

import numpy as np
import pytest
import torch

from asc_cpp_b200._abi import PLAN_TRANSPOSE, FormatKind, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import (CsrPlan, CudaConvertCompressed, CudaConvertCoordinates,
                                      CudaSpmv)

from gpu_util import bits_equal, context, csr, dev, host, vec

pytestmark = pytest.mark.gpu


def bucket_offsets(keys, limit):
    return np.concatenate([[0], np.cumsum(np.bincount(keys, minlength=limit))]).astype(np.int64)


def values(rng, n, dt):
    v = rng.standard_normal(n)
    return (v + 1j * rng.standard_normal(n)).astype(dt) if np.dtype(dt).kind == "c" else \
        v.astype(dt)


@pytest.mark.parametrize("n,rows,cols", [
    (1, 1, 1), (31, 16, 2), (4095, 70, 300), (4096, 5000, 256), (4097, 20, 257),
    (20_000, 100_000, 3), (70_001, 900, 70_000), (50_000, 40, 20_000_000),
    (9_000, 77, 1 << 33),  # 64-bit words
])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex128])
def test_coordinates_to_csr_at_sort_edges(cuda_lib, n, rows, cols, dt):
    rng = np.random.default_rng(n + rows)
    coo = np.stack([rng.integers(0, rows, n), rng.integers(0, cols, n)], 1).astype(np.int64)
    val = values(rng, n, dt)
    ctx = context()
    for fmt, k in ((FormatKind.kCsr, 0), (FormatKind.kCsc, 1)):
        limit = (rows, cols)[k]
        if limit > 1 << 25:
            continue  # the offsets alone would take the test's time
        m = CudaConvertCoordinates(ctx, rows, cols, dev(coo), dev(val), fmt)
        order = np.argsort(coo[:, k], kind="stable")
        assert bits_equal(host(m.offsets), bucket_offsets(coo[:, k], limit))
        assert bits_equal(host(m.indices), coo[order, 1 - k])
        assert bits_equal(host(m.values), val[order])
    ctx.close()


@pytest.mark.parametrize("lengths,cols", [
    ([0, 0, 5, 0, 4091, 0, 1, 0], 5000),      # rows that end at a tile's end
    ([4096], 4097), ([1] * 4097, 9),
    ([0] * 9000 + [3] + [0] * 9000, 4),       # far more rows than entries
    ([2000, 0, 0, 3000] * 5 + [0] * 4096, 3001),
])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64])
def test_transposed_structure_at_tile_edges(cuda_lib, lengths, cols, dt):
    rng = np.random.default_rng(len(lengths))
    rows = len(lengths)
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.permutation(cols)[:n]) for n in lengths]).astype(np.int64)
    val = values(rng, idx.size, dt)
    ctx = context()
    a = csr(rows, cols, ptr, idx, val)
    t = CudaConvertCompressed(ctx, a)
    order = np.argsort(idx, kind="stable")
    row_of = np.repeat(np.arange(rows), lengths)
    assert bits_equal(host(t.offsets), bucket_offsets(idx, cols))
    assert bits_equal(host(t.indices), row_of[order])
    assert bits_equal(host(t.values), val[order])
    # with the permutation (a plan) and without (a plain call): the same product
    x = dev(values(rng, rows, dt))
    y0 = dev(values(rng, cols, dt))
    plan = CsrPlan(ctx, a, PLAN_TRANSPOSE)
    got = []
    for p in (None, plan):
        y = y0.clone()
        CudaSpmv(ctx, SparseBlasTranspose.kTranspose, 0.5, a, vec(x, writable=False), vec(y),
                 plan=p)
        got.append(host(y))
    assert bits_equal(*got)
    plan.close()
    ctx.close()
    torch.cuda.synchronize()
