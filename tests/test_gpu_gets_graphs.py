"""Large batches of gets recorded into CUDA graphs (VoxTree::get, voxtree.rs:145-159): reads write nothing but their
outputs, so graphs of different sizes may be replayed side by side on several streams."""
import ctypes as C

import numpy as np
import pytest

from voxelis_gb300 import workloads as W
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
def test_graphs_of_gets_side_by_side(gpu_lib):
    import torch

    depth, sizes = 6, (1 << 20, 1 << 22, (1 << 21) + 1)
    it = VoxInterner(64 << 20, lib=gpu_lib)
    tree = VoxTree(depth)
    grid = W.dune_world_chunks(1, 1, depth=depth, seed=4)
    it.build_dense([tree], grid)
    capture = torch.cuda.Stream()
    it.set_stream(capture.cuda_stream)
    rng = np.random.default_rng(0)
    work = []
    for n in sizes:
        xyz = rng.integers(0, 1 << depth, (n, 3)).astype(np.int32)
        want = torch.from_numpy(grid[0][xyz[:, 1], xyz[:, 2], xyz[:, 0]]).cuda()
        arrays = [torch.full((n,), tree.tree, dtype=torch.int32, device="cuda"), torch.from_numpy(xyz).cuda(),
                  torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        before = gpu_lib.kernel_launches()
        with torch.cuda.graph(graph, stream=capture):
            it._call("get_many_async", C.c_uint64(n), *(C.c_void_p(a.data_ptr()) for a in arrays))
        assert gpu_lib.kernel_launches() - before == 1  # the reads alone: no kernel that fills a shared table
        work.append((graph, arrays, want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    for _ in range(4):
        for graph, arrays, _, stream in work:
            with torch.cuda.stream(stream):
                graph.replay()
        torch.cuda.synchronize()
        for _, (_, _, found, values), want, _ in work:
            assert torch.equal(values, want) and torch.equal(found.bool(), want != 0)
            found.zero_(), values.zero_()
        torch.cuda.synchronize()
    it.sync()
    it.set_stream(0)
