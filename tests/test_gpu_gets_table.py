"""Large batches of gets, which start from a table of upper nodes (VoxTree::get, voxtree.rs:145-159;
get_at_depth, utils/common.rs:122-156): trees of several depths in one interner, among them trees shallower
than the table, EMPTY ones, single leaves and freed handles; positions on and outside the edges; and a second
call after edits, which must see them."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_E_INVALID_ARG, VX_E_OOB, VX_PATCH_P1, VX_PATCH_P2, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("bits,depths,n", [
    (8, (1, 2, 3, 4, 5, 6), 1 << 19), (16, (8,), 1 << 19), (8, (5,) * 300, (1 << 19) + 3), (8, (7, 0, 3), (1 << 20) + 1),
    (16, (4, 2), (1 << 19) - 1),
])
def test_gets_equal_the_dense_trees(gpu_lib, bits, depths, n):
    rng = np.random.default_rng(len(depths) + bits)
    it = VoxInterner(256 << 20, bits, VX_PATCH_P1 | VX_PATCH_P2, lib=gpu_lib)
    trees = [VoxTree(d) for d in depths]
    spare = VoxTree(3)
    handles = np.array([t._bind(it) for t in trees], np.uint32)
    spare.fill(it, 9)
    for k, (t, d) in enumerate(zip(trees, depths)):
        if k % 7 == 5:
            continue  # EMPTY
        if d < 2 or k % 7 == 4:
            t.fill(it, 1 + k % 5)
        else:
            side = 1 << d
            g = rng.integers(0, 4, (side // 2,) * 3).repeat(2, 0).repeat(2, 1).repeat(2, 2).astype(it.dtype)
            g[: side // 2] = rng.integers(0, 300 if bits == 16 else 200)
            it.build_dense([t], g[None])
    for step in range(2):
        dense = [t.to_vec(it) if d else None for t, d in zip(trees, depths)]
        which = rng.integers(0, len(trees), n)
        side = np.array([1 << d for d in depths])[which]
        xyz = (rng.random((n, 3)) * side[:, None]).astype(np.int32)
        edge = rng.random((n, 3)) < 0.1
        xyz = np.where(edge, side[:, None] - 1, xyz).astype(np.int32)
        found, values = it.get_many(handles[which], xyz)
        want = np.zeros(n, it.dtype)
        for k, g in enumerate(dense):
            sel = which == k
            p = xyz[sel]
            want[sel] = g[p[:, 1], p[:, 2], p[:, 0]] if g is not None else (trees[k].get(it, (0, 0, 0)) or 0)
        np.testing.assert_array_equal(values, want)
        np.testing.assert_array_equal(found, want != 0)
        for t, d in zip(trees, depths):
            if d:
                t.set(it, (1, 0, 1), 7)
    # a position outside a tree, and a freed handle
    out = xyz.copy()
    out[n // 2, 2] = side[n // 2]
    with pytest.raises(VoxelisError) as e:
        it.get_many(handles[which], out)
    assert e.value.status == VX_E_OOB
    freed = handles[which].copy()
    freed[n // 3] = spare.tree
    it.lib.call("tree_destroy", it.handle, spare.tree, handle=it.handle)
    with pytest.raises(VoxelisError) as e:
        it.get_many(freed, np.zeros((n, 3), np.int32))
    assert e.value.status == VX_E_INVALID_ARG
