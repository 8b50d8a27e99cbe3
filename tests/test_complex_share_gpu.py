"""Complex contracted SpMV where several lanes share a row: 1 to 32 of them, rows
shorter than their lanes, rows that end inside and on a round, a last warp that is
not full."""

import numpy as np
import pytest
import torch

from asc_cpp_b200._abi import Determinism, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import CudaCsrArray, CudaSpmv

from gpu_util import context, dev, gamma, host, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
@pytest.mark.parametrize("per_warp", [1, 2, 3, 5, 9, 17, 33])
def test_shared_rows(cuda_lib, dt, per_warp):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, cols = sms * 16 * per_warp + 7, 4000  # `per_warp` rows to each of 16 warps an SM
    rng = np.random.default_rng(per_warp)
    lengths = rng.integers(0, 12, rows)
    lengths[::97] = rng.choice([31, 32, 33, 127, 128, 129, 256, 300], lengths[::97].size)
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = rng.integers(0, cols, ptr[-1])

    def values(n):
        return (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)).astype(dt)

    val, x, y0, alpha = values(idx.size), values(cols), values(rows), 0.75 - 0.5j
    ctx = context(Determinism.kBackendDefault)
    y = dev(y0)
    CudaSpmv(ctx, SparseBlasTranspose.kNone, alpha, CudaCsrArray(rows, cols, dev(ptr), dev(idx), dev(val)),
             vec(dev(x), cols, 1, writable=False), vec(y, rows, 1))
    got = host(y)
    ctx.close()
    wide = np.zeros(rows, np.complex128)
    size = np.zeros(rows)
    row = np.repeat(np.arange(rows), lengths)
    terms = val.astype(np.complex128) * x.astype(np.complex128)[idx]
    np.add.at(wide, row, terms)
    np.add.at(size, row, np.abs(terms))
    # a complex product and sum round at most 4 times per component
    real = np.float64 if dt == np.complex128 else np.float32
    bound = gamma(4 * lengths + 8, real) * (2 * abs(alpha) * size + 2 * np.abs(y0.astype(np.complex128)))
    assert np.all(np.abs(got - (y0 + alpha * wide)) <= bound + 1e-30)
    assert np.array_equal(got[lengths == 0].view(real), y0[lengths == 0].view(real))
