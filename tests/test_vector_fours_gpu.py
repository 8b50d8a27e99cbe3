"""The vector SpMV kernel in aligned fours: rows that begin and end anywhere in a
four, the last row at the very end of the arrays, empty and long rows, arrays
off 32-byte boundaries (single loads), strides."""

import numpy as np
import pytest
import torch

from asc_cpp_b200 import synthetic
from asc_cpp_b200._abi import Determinism, Variant
from asc_cpp_b200.sparse_cuda import CsrPlan, CudaCsrArray

from gpu_util import assert_within_bound, context, dev, host, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("lanes", [1, 2, 4])
@pytest.mark.parametrize("rows,most,shift", [(1, 70, 0), (333, 110, 0), (333, 110, 1), (40, 5, 0)])
@pytest.mark.parametrize("incx,incy,beta", [(1, 1, 0.5), (2, 3, 0.0)])
def test_vector_fours(cuda_lib, restatement, dt, lanes, rows, most, shift, incx, incy, beta):
    rng = np.random.default_rng(rows + lanes)
    a_h = synthetic.random_csr(rng, rows, 500, most, dt, 0.1)
    idx, val = (torch.zeros(a_h.nnz + 4, dtype=t, device="cuda")[shift:shift + a_h.nnz]
                for t in (torch.int64, dev(a_h.val).dtype))
    idx.copy_(dev(a_h.idx))
    val.copy_(dev(a_h.val))
    a = CudaCsrArray(rows, 500, dev(a_h.ptr), idx, val)
    x, y0 = rng.uniform(-1, 1, 500).astype(dt), rng.uniform(-1, 1, rows).astype(dt)
    xd, yd = np.zeros(500 * incx, dt), np.full(rows * incy, 7, dt)
    xd[::incx], yd[::incy] = x, y0
    ctx = context(Determinism.kBackendDefault)
    ctx.set_variant(Variant.kVector, lanes)
    plan = CsrPlan(ctx, a)
    y = dev(yd)
    plan.csr_spmv(-1.5, vec(dev(xd), 500, incx, writable=False), beta, vec(y, rows, incy))
    got = host(y)
    exact, absval = restatement.extended(0, rows, 500, a_h.ptr, a_h.idx, a_h.val, x)
    assert_within_bound(got[::incy], exact, absval, np.diff(a_h.ptr), dt, -1.5,
                        np.abs(beta * y0.astype(np.float64)),
                        -1.5 * exact + beta * y0.astype(np.longdouble))
    kept = np.ones(rows * incy, bool)
    kept[::incy] = False
    assert (got[kept] == 7).all()
    plan.close()
    ctx.close()
