"""Tile bounds of the segmented SpMV kernel: found by the kernel itself up to
one tile per resident warp, by the partition kernel beyond; and the batch's
tiles -- matrix search over more than 32 x 32 matrices with empty ones among
them, arrays on 16- but not 32-byte boundaries, tiles of more than 32 rows."""

import numpy as np
import pytest
import torch

from asc_cpp_b200 import synthetic
from asc_cpp_b200._abi import Determinism
from asc_cpp_b200.sparse_cuda import (CsrPlan, CudaBatch, CudaCsrArray, CudaCsrSpmv,
                                      CudaCsrSpmvWorkspaceSize, CudaStridedVectorView)

from gpu_util import assert_within_bound, bits_equal, context, csr, dev, host, vec

pytestmark = pytest.mark.gpu


def one_pass_rows():
    """Rows of one entry each (3 items a row, 251 a tile) that give every warp
    of a 6-CTA-per-SM grid one tile."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms * 6 * 4 * 251 // 3


@pytest.mark.parametrize("extra", [-84, -1, 0, 1, 84])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_bounds_search_at_the_one_pass_limit(cuda_lib, restatement, extra, dt):
    rows = one_pass_rows() + extra
    rng = np.random.default_rng(rows)
    lengths = np.ones(rows, np.int64)
    lengths[rng.integers(0, rows, 40)] = 0
    lengths[rows // 3] = 700  # a row past its tile's window
    lengths[-1] = 2
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = np.concatenate([rng.integers(0, rows, ptr[rows // 3]),
                          np.sort(rng.permutation(rows)[:700]),
                          rng.integers(0, rows - 1, ptr[-1] - ptr[rows // 3] - 700)])
    idx[-2:] = [rows - 2, rows - 1]
    val = rng.standard_normal(idx.size).astype(dt)
    x, y0 = rng.uniform(-1, 1, rows).astype(dt), rng.uniform(-1, 1, rows).astype(dt)
    expect = y0.copy()
    restatement.compat_spmv(ptr, idx.astype(np.int64), val, 1.5, x, 0.5, expect)
    ctx = context()
    a = csr(rows, rows, ptr, idx, val)
    xv = vec(dev(x), writable=False)
    plain, planned = dev(y0), dev(y0)
    need = CudaCsrSpmvWorkspaceSize(ctx, a, xv, vec(plain))
    CudaCsrSpmv(ctx, 1.5, a, xv, 0.5, vec(plain),
                torch.empty(max(need, 1), dtype=torch.uint8, device="cuda"))
    plan = CsrPlan(ctx, a)
    plan.csr_spmv(1.5, xv, 0.5, vec(planned))
    assert bits_equal(host(plain), expect)
    assert bits_equal(host(planned), expect)
    plan.close()
    ctx.close()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shift", [0, 16, 8])  # bytes past a 32-byte boundary
@pytest.mark.parametrize("mode", [Determinism.kDeterministic, Determinism.kBackendDefault])
def test_batch_tiles(cuda_lib, restatement, dt, shift, mode):
    rng = np.random.default_rng(shift)
    count = 1500
    mats = []
    for i in range(count):
        rows = int(rng.integers(0, 60)) if i % 7 else 0
        if i in (5, 1400):
            rows = 900
        if rows == 0:
            mats.append(synthetic.Csr(0, 3, np.zeros(1, np.int64), np.zeros(0, np.int64),
                                      np.zeros(0, dt)))
        else:
            mats.append(synthetic.random_csr(rng, rows, max(rows, 4), 4 if i != 5 else 800, dt, 0.2))
    es = np.dtype(dt).itemsize
    pad = 32  # every matrix's entries begin `shift` bytes past a 32-byte boundary
    total = sum((m.nnz * 8 + 2 * pad) // pad * pad // 8 + pad for m in mats) + pad
    idx, val = torch.zeros(total, dtype=torch.int64, device="cuda"), torch.zeros(
        total, dtype=torch.from_numpy(np.zeros(1, dt)).dtype, device="cuda")
    arrays, xs, ys, at, host_x, host_y = [], [], [], 0, [], []
    for m in mats:
        i0, v0 = at + shift // 8, at + max(shift // es, 0)
        idx[i0:i0 + m.nnz] = dev(m.idx)
        val[v0:v0 + m.nnz] = dev(m.val)
        arrays.append(CudaCsrArray(m.rows, m.cols, dev(m.ptr), idx[i0:i0 + m.nnz],
                                   val[v0:v0 + m.nnz]))
        at += (m.nnz + 8 + 7) // 8 * 8
        hx, hy = rng.uniform(-1, 1, m.cols).astype(dt), rng.uniform(-1, 1, m.rows).astype(dt)
        host_x.append(hx)
        host_y.append(hy)
        xs.append(CudaStridedVectorView.of(dev(hx), False))
        ys.append(CudaStridedVectorView.of(dev(hy) if m.rows else dev(np.zeros(1, dt))[:0]))
    ctx = context(mode)
    batch = CudaBatch(ctx, arrays, xs, ys)
    batch.spmv(-1.5, 0.5)
    torch.cuda.synchronize()
    for m, hx, hy, y in zip(mats, host_x, host_y, ys):
        if m.rows == 0:
            continue
        got = host(y.tensor)
        if mode == Determinism.kDeterministic:
            expect = hy.copy()
            restatement.compat_spmv(m.ptr, m.idx, m.val, -1.5, hx, 0.5, expect)
            assert bits_equal(got, expect)
        else:
            exact, absval = restatement.extended(0, m.rows, m.cols, m.ptr, m.idx, m.val, hx)
            assert_within_bound(got, exact, absval, np.diff(m.ptr), dt, -1.5,
                                np.abs(0.5 * hy.astype(np.float64)),
                                -1.5 * exact + 0.5 * hy.astype(np.longdouble))
    batch.close()
    ctx.close()
