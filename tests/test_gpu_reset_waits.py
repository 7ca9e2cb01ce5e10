"""vx_interner_reset returns when the work queued before it is done: a program may then free or refill the device buffers
of its asynchronous calls."""
import ctypes as C

import numpy as np
import pytest

from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
def test_reset_waits_for_queued_work(gpu_lib):
    import torch

    it = VoxInterner(64 << 20, lib=gpu_lib)
    stream = torch.cuda.Stream()
    it.set_stream(stream.cuda_stream)
    tree = VoxTree(5)
    it.build_dense([tree], np.full((1, 32, 32, 32), 2, np.uint8))
    n = 1 << 24
    trees = torch.full((n,), tree.tree, dtype=torch.int32, device="cuda")
    xyz = torch.randint(0, 32, (n, 3), dtype=torch.int32, device="cuda")
    found = torch.zeros(n, dtype=torch.uint8, device="cuda")
    values = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        for _ in range(40):  # some milliseconds of reads
            it._call("get_many_async", C.c_uint64(n), *(C.c_void_p(a.data_ptr()) for a in (trees, xyz, found, values)))
        queued = stream.record_event()
        it._call("interner_reset")
        assert queued.query()
    assert it.stats()["alive_nodes"] == 1
    it.set_stream(0)
