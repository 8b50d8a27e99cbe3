"""A batch's schedule as it is launched: tiles per grab that were set are taken as
they are, and only those that nobody set give way to a small batch."""

import numpy as np
import pytest
import torch

from asc_cpp_b200.sparse_cuda import CudaBatch, CudaCsrArray, SparseCudaContext

from gpu_util import bits_equal, host, vec

pytestmark = pytest.mark.gpu


def kernel_grids(graph):
    """Blocks of each kernel node of a captured graph."""
    from cuda.bindings import driver
    handle = driver.CUgraph(graph.raw_cuda_graph())
    rc, nodes, count = driver.cuGraphGetNodes(handle, 0)
    assert rc == driver.CUresult.CUDA_SUCCESS
    rc, nodes, count = driver.cuGraphGetNodes(handle, count)
    assert rc == driver.CUresult.CUDA_SUCCESS
    grids = []
    for node in nodes[:count]:
        rc, kind = driver.cuGraphNodeGetType(node)
        if kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            rc, params = driver.cuGraphKernelNodeGetParams(node)
            assert rc == driver.CUresult.CUDA_SUCCESS
            grids.append(params.gridDimX)
    return grids


@pytest.mark.parametrize("chunk", [None, 4, 32])
def test_chunk_is_the_one_that_was_set(cuda_lib, chunk):
    rows, per, count = 512, 8, 40
    rng = np.random.default_rng(7)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = SparseCudaContext.Create(0, stream=stream)
        ptr = torch.arange(rows + 1, device="cuda") * per
        matrices, xs, ys = [], [], []
        for _ in range(count):
            idx = np.sort(rng.integers(0, rows, (rows, per)), 1).reshape(-1)
            matrices.append(CudaCsrArray(rows, rows, ptr, torch.from_numpy(idx).cuda(),
                                         torch.from_numpy(rng.standard_normal(idx.size)).cuda()))
            xs.append(torch.from_numpy(rng.standard_normal(rows)).cuda())
            ys.append(torch.zeros(rows, dtype=torch.float64, device="cuda"))
        batch = CudaBatch(ctx, matrices, [vec(x, writable=False) for x in xs],
                          [vec(y) for y in ys])
        batch.spmv(1.0, 0.0)
        expect = [host(y).copy() for y in ys]
        if chunk is not None:
            batch.set_schedule(chunk)
            assert batch.schedule() == (chunk, 0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        batch.spmv(1.0, 0.0)
    # 512 rows of 8 entries: 16 to 32 tiles of 256 items a matrix, 640 to 1280 in
    # all, fewer than there are resident warps (four a block)
    grids = kernel_grids(graph)
    assert len(grids) == 1
    if chunk is None:
        assert grids[0] >= 16 * count // 4
    else:
        assert 16 * count // (4 * chunk) <= grids[0] <= 32 * count // (4 * chunk) + 1
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    assert all(bits_equal(host(y), e) for y, e in zip(ys, expect))
    del graph
    batch.close()
    ctx.close()
