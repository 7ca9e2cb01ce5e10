"""Batched occupancy masks of builders with more trees than the kernel lists side by side (64), none, and a few, and of
trees that lie outside of their builder: the masks of one call per builder (utils/mesh.rs:418-597)."""
import numpy as np
import pytest

import torch
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("depth,per_builder", [(1, (300, 0, 5)), (2, (64, 65, 129)), (3, (63, 200, 1)), (4, (64, 17, 0))])
def test_many_trees_a_builder(gpu_lib, depth, per_builder):
    import ctypes as C

    rng = np.random.default_rng(depth)
    side, n, slots = 1 << depth, sum(per_builder), 4
    it = VoxInterner(64 << 20, 8, 0, lib=gpu_lib)
    trees = [VoxTree(depth) for _ in range(n)]
    for t in trees:
        for _ in range(3):
            t.set(it, rng.integers(0, side, 3), int(rng.integers(1, 4)))
    builder = np.repeat(np.arange(3), per_builder)
    cells = [rng.permutation((64 // side) ** 3)[:k] for k in per_builder]
    at = np.concatenate(cells)
    c = 64 // side
    offsets = (np.stack([at % c, at // c % c, at // (c * c)], 1) * side).astype(np.int32)
    order = rng.permutation(n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()  # noqa: E731
    z = lambda *shape, dtype=torch.int64: torch.zeros(shape, dtype=dtype, device="cuda")  # noqa: E731
    planes = 3 * 64 * 64
    glob, active, count = z(3, planes), z(3, 6), z(3, dtype=torch.int32)
    ids, counts, masks = z(3, slots, dtype=torch.int32), z(3, slots), z(3, slots, planes)
    handles = np.array([t.tree for t in trees], np.uint32)[order]
    args = [dev(handles), dev(builder[order].astype(np.int32)), dev(offsets[order])]
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    gpu_lib.call("occupancy_masks_async", it.handle, 3, n, *[P(a) for a in args], depth, slots, P(glob), P(active), P(count),
                 P(ids), P(counts), P(masks), handle=it.handle)
    it.sync()
    for b in range(3):
        mine = np.flatnonzero(builder == b)
        if not len(mine):
            assert int(count[b]) == 0 and not glob[b].any() and not masks[b].any()
            continue
        want = it.occupancy_masks([trees[k] for k in mine], offsets[mine].astype(np.uint32), slots)
        np.testing.assert_array_equal(glob[b].cpu().numpy().view(np.uint64), want["global"].reshape(-1))
        np.testing.assert_array_equal(active[b].cpu().numpy().view(np.uint64), want["active"])
        assert int(count[b]) == len(want["materials"])
        for k, (m, (number, plane)) in enumerate(sorted(want["materials"].items())):
            assert int(ids[b, k]) == m and int(counts[b, k]) == number
            np.testing.assert_array_equal(masks[b, k].cpu().numpy().view(np.uint64), plane.reshape(-1))
