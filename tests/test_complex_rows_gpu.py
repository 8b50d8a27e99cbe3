"""Complex SpMV where its rounds of 128 entries can go wrong: rows that end on a
round's end, rows of several rounds one behind the other, empty rows, more rows
than a warp takes, arrays off whole-element boundaries, strided vectors."""

import numpy as np
import pytest
import torch

from asc_cpp_b200 import synthetic
from asc_cpp_b200._abi import Determinism, SparseBlasTranspose
from asc_cpp_b200.sparse_cuda import CudaCsrArray, CudaSpmv
from oracle import CSR, OP_NONE

from gpu_util import bits_equal, context, dev, gamma, host, vec

pytestmark = pytest.mark.gpu

SHAPES = [
    [128, 128, 256, 384, 1, 0, 127], [0, 0, 640, 512, 3], [1], [129, 0, 1, 1], [5] * 20_000,
    [27] * 9000 + [2000, 0, 4096, 128], [300] * 40,
]


@pytest.mark.parametrize("lengths", SHAPES, ids=range(len(SHAPES)))
@pytest.mark.parametrize("dt", [np.complex64, np.complex128])
@pytest.mark.parametrize("shift,incx,incy", [(0, 1, 1), (1, 1, 1), (0, 2, 3)])
def test_complex_rows(cuda_lib, restatement, lengths, dt, shift, incx, incy):
    rng = np.random.default_rng(len(lengths))
    rows, cols = len(lengths), max(5000, max(lengths))
    ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    idx = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) if n > 50 else
                          np.sort(rng.integers(0, cols, n)) for n in lengths]).astype(np.int64)

    def values(n):
        return (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)).astype(dt)

    val, x, y0 = values(idx.size), values(cols), values(rows)
    alpha = 0.75 - 0.5j
    # `shift` components past a whole-element boundary
    real = np.dtype(dt).itemsize // 2
    room = torch.zeros((idx.size + 2) * 2 * real, dtype=torch.uint8, device="cuda")
    stored = room[shift * real:shift * real + idx.size * 2 * real]
    stored.copy_(dev(val).view(torch.uint8))
    if shift and real == 4:
        pytest.skip("complex64 arrays start on 8-byte boundaries")
    a = CudaCsrArray(rows, cols, dev(ptr), dev(idx), stored.view(torch.complex128 if real == 8 else
                                                                 torch.complex64)
                     if not shift else _Raw(stored, idx.size))
    xd, yd = values(cols * incx), values(rows * incy)
    xd[::incx], yd[::incy] = x, y0
    for mode in (Determinism.kDeterministic, Determinism.kBackendDefault):
        ctx = context(mode)
        y = dev(yd)
        CudaSpmv(ctx, SparseBlasTranspose.kNone, alpha, a,
                 vec(dev(xd), cols, incx, writable=False), vec(y, rows, incy))
        got = host(y)[::incy]
        ctx.close()
        expect = y0.copy()
        restatement.standard_spmv(CSR, OP_NONE, rows, cols, ptr, idx, val, alpha, x, expect)
        if mode == Determinism.kDeterministic:
            assert bits_equal(got, expect)
        else:
            wide = np.zeros(rows, np.complex128)
            size = np.zeros(rows)
            row = np.repeat(np.arange(rows), lengths)
            terms = val.astype(np.complex128) * x.astype(np.complex128)[idx]
            np.add.at(wide, row, terms)
            np.add.at(size, row, np.abs(terms))
            # a complex product and sum round at most 4 times per component
            bound = gamma(4 * np.asarray(lengths) + 8, np.float64 if real == 8 else np.float32) * (
                2 * abs(alpha) * size + 2 * np.abs(y0.astype(np.complex128)))
            assert np.all(np.abs(got - (y0 + alpha * wide)) <= bound + 1e-30)


class _Raw:
    """A byte tensor seen as complex128 elements off a 16-byte boundary (torch
    has no such view)."""

    def __init__(self, data, n):
        self.data, self.n, self.dtype, self.is_cuda = data, n, torch.complex128, True

    def data_ptr(self):
        return self.data.data_ptr()

    def numel(self):
        return self.n
