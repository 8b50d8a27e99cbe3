"""Triangular solves in row order of matrices that are stored whole, one
right-hand side: batches of entries that hold the diagonal only, entries of the
other triangle only, or nothing but those at a row's start or end, for rows of up
to 4 entries and beyond (batches of 3 and of 2); every lane of a group in its own
place.  DETERMINISTIC, bit for bit; BACKEND_DEFAULT repeats bit for bit."""

import numpy as np
import pytest

from asc_cpp_b200._abi import (Determinism, SparseBlasDiagonal, SparseBlasLayout,
                               SparseBlasTranspose, SparseBlasTriangle)
from asc_cpp_b200.sparse_cuda import CudaSparseTriangularSolveMultiple, DenseMatrixView

from gpu_util import bits_equal, context, csr, dev, host

pytestmark = pytest.mark.gpu

N = 1000


def whole(dt, most, seed):
    """Rows of 1 to `most` entries on both sides of the diagonal, near and far;
    every seventh row lies in one triangle only."""
    rng = np.random.default_rng(seed)
    rows = []
    for r in range(N):
        n = rng.integers(0, most)
        near = r + rng.integers(-4, 5, n)
        far = rng.integers(0, N, n)
        c = np.where(rng.random(n) < 0.6, near, far)
        c = c[(c >= 0) & (c < N)]
        if r % 7 == 3:
            c = c[c > r]
        if r % 7 == 5:
            c = c[c < r]
        rows.append(np.unique(np.append(c, r)))
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.int64)
    idx = np.concatenate(rows).astype(np.int64)
    val = rng.uniform(-1, 1, idx.size) / most
    if np.iscomplexobj(dt(0)):
        val = val + 1j * rng.uniform(-1, 1, idx.size) / most
    val[idx == np.repeat(np.arange(N), np.diff(ptr))] += 1.5
    b = rng.uniform(-1, 1, N) + (0.5j if np.iscomplexobj(dt(0)) else 0)
    return ptr, idx, val.astype(dt), b.astype(dt)


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("most", [3, 8, 12, 40])
@pytest.mark.parametrize("diag", list(SparseBlasDiagonal))
def test_whole_matrix_in_row_order(cuda_lib, restatement, dt, most, diag):
    ptr, idx, val, b = whole(dt, most, most)
    assert (idx.size <= 4 * N) == (most <= 8)
    a = csr(N, N, ptr, idx, val)
    for tri in SparseBlasTriangle:
        for op in (SparseBlasTranspose.kNone, SparseBlasTranspose.kConjugateTranspose):
            want = restatement.triangular_solve(int(op), int(tri), int(diag), N, ptr, idx, val, 1.25,
                                                b, 1, None, 1)
            fast = []
            for mode in (Determinism.kDeterministic, Determinism.kBackendDefault,
                         Determinism.kBackendDefault):
                ctx = context(mode)
                x = dev(b)
                CudaSparseTriangularSolveMultiple(ctx, op, 1.25, a, tri, diag,
                                                  DenseMatrixView(x, N, 1, SparseBlasLayout(1)))
                ctx.synchronize()
                assert ctx.device_status() == 0
                got = host(x)
                ctx.close()
                if mode == Determinism.kDeterministic:
                    assert bits_equal(got, want), (tri, op)
                else:
                    fast.append(got)
            assert bits_equal(*fast), (tri, op)
