"""Batched occupancy masks against one call per builder: every depth, more and fewer materials than planes
and than slots, overlapping trees at offsets that are no multiple of anything, outputs that are only
8-byte aligned, and a builder without trees (vx_occupancy_masks_async, utils/mesh.rs:418-597)."""
import ctypes as C

import numpy as np
import pytest

from voxelis_gb300._abi import VX_E_OOB, VX_PATCH_P1, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree

PLANES = 3 * 4096


def batched(it, handles, builder_of, offsets, n_builders, depth, slots, shift=0):
    """The batched call; shift: words that the outputs start past a 16-byte boundary."""
    import torch

    def out(n, dtype):
        t = torch.full((n + 2,), -1, dtype=dtype, device="cuda")  # every word has to be written
        return t, C.c_void_p(t.data_ptr() + 8 * shift)

    T = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()  # noqa: E731
    t, b, o = T(handles), T(builder_of), T(offsets.ravel())
    glob, gp = out(n_builders * PLANES, torch.int64)
    masks, mp = out(n_builders * slots * PLANES, torch.int64)
    act = torch.full((n_builders * 6,), -1, dtype=torch.int64, device="cuda")
    nm = torch.full((n_builders,), -1, dtype=torch.int32, device="cuda")
    ids = torch.zeros(n_builders * slots, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(n_builders * slots, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    P = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    it._call("occupancy_masks_async", n_builders, len(handles), P(t), P(b), P(o), depth, slots, gp, P(act), P(nm), P(ids),
             P(cnt), mp)
    it.sync()
    H = lambda x, n: x.cpu().numpy()[shift:shift + n].view(np.uint64)  # noqa: E731
    return (H(glob, n_builders * PLANES).reshape(n_builders, 3, 64, 64), act.cpu().numpy().view(np.uint64).reshape(-1, 6),
            nm.cpu().numpy(), ids.cpu().numpy().reshape(n_builders, slots), cnt.cpu().numpy().reshape(n_builders, slots),
            H(masks, n_builders * slots * PLANES).reshape(n_builders, slots, 3, 64, 64))


@pytest.mark.gpu
@pytest.mark.parametrize("depth,materials,slots,shift", [
    (1, 2, 4, 0), (2, 1, 1, 0), (3, 3, 8, 1), (4, 4, 4, 0), (4, 200, 256, 0), (5, 7, 3, 0), (5, 3, 2, 1), (6, 2, 3, 0),
])
def test_batched_masks_equal_one_call_per_builder(gpu_lib, depth, materials, slots, shift):
    rng = np.random.default_rng(100 * depth + materials)
    side, n_builders = 1 << depth, 4
    n = 9 if depth < 6 else 4
    it = VoxInterner(256 << 20, 8, VX_PATCH_P1, lib=gpu_lib)
    trees = [VoxTree(depth) for _ in range(n)]
    if depth == 1:  # batches and dense builds need MaxDepth 2
        for k, t in enumerate(trees):
            t.fill(it, 1 + k % materials)
            t.set(it, (k & 1, 1, 0), 1 + (k + 1) % materials)
            if k % 3:
                t.set(it, (0, 0, 1), 0)
    else:
        grids = rng.integers(1, materials + 1, (n, side, side, side)).astype(np.uint8)
        grids[rng.random(grids.shape) < 0.4] = 0
        grids[:, : side // 2] = grids[:, :1, :1, :1]  # uniform halves
        it.build_dense(trees, grids)
    handles = np.array([t._bind(it) for t in trees], np.uint32)
    builder_of = np.sort(rng.integers(0, n_builders - 1, n)).astype(np.uint32)  # the last one stays empty
    rng.shuffle(builder_of)
    offsets = rng.integers(0, 64 - side + 1, (n, 3)).astype(np.uint32)
    glob, act, nm, ids, cnt, masks = batched(it, handles, builder_of, offsets, n_builders, depth, slots, shift)
    for b in range(n_builders):
        sel = np.flatnonzero(builder_of == b)
        if not len(sel):
            assert nm[b] == 0 and not glob[b].any() and not act[b].any() and not masks[b].any()
            continue
        one = it.occupancy_masks([trees[k] for k in sel], offsets[sel])
        np.testing.assert_array_equal(glob[b], one["global"])
        np.testing.assert_array_equal(act[b], one["active"])
        mats = sorted(one["materials"])
        assert nm[b] == len(mats)
        for k, m in enumerate(mats[:slots]):
            assert ids[b, k] == m and cnt[b, k] == one["materials"][m][0]
            np.testing.assert_array_equal(masks[b, k], one["materials"][m][1])
        assert not masks[b, len(mats):].any()


@pytest.mark.gpu
def test_tree_outside_its_builder_is_refused(gpu_lib):
    it = VoxInterner(64 << 20, 8, VX_PATCH_P1, lib=gpu_lib)
    tree = VoxTree(4)
    it.build_dense([tree], np.full((1, 16, 16, 16), 5, np.uint8))
    handles = np.array([tree._bind(it)] * 2, np.uint32)
    for builder_of, offsets in (([0, 7], [[0, 0, 0], [0, 0, 0]]), ([0, 0], [[0, 0, 0], [49, 0, 0]])):
        with pytest.raises(VoxelisError) as e:
            batched(it, handles, np.array(builder_of, np.uint32), np.array(offsets, np.uint32), 1, 4, 2)
        assert e.value.status == VX_E_OOB
