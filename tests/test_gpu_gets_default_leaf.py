"""Batched gets of voxels under a leaf of the default value, which a batch's fill of 0 leaves (voxtree.rs:742-758): met
above the tree's depth it is a voxel of value 0, as get_at_depth has it (utils/common.rs:122-156). On both sides of
the size from which gets start from a table of upper nodes, for trees as deep as the table, deeper and shallower."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P2
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1 << 12, (1 << 20) - 1, 1 << 20, 1 << 22])
@pytest.mark.parametrize("depths", [(2,), (5,), (6,), (7,), (0, 1, 2, 3), (4, 2) * 200])
def test_gets_under_a_default_leaf(oracle_lib, gpu_lib, n, depths):
    its, handles = [], []
    for lib in (oracle_lib, gpu_lib):
        rng = np.random.default_rng(len(depths))
        it = VoxInterner(64 << 20, 8, VX_PATCH_P1 | VX_PATCH_P2, lib=lib)
        trees = [VoxTree(d) for d in depths]
        handles.append(np.array([t._bind(it) for t in trees], np.uint32))
        for k, (t, d) in enumerate(zip(trees, depths)):
            if d < 2:
                t.fill(it, 3)
                continue
            b = t.create_batch(it)
            b.fill(it, 0)
            if k % 3 < 2:  # (every third tree stays one leaf)
                xyz = rng.integers(0, 1 << d, (2, 3)).astype(np.int32)
                b.set_many(xyz, np.array([5, 6], np.uint32))
            t.apply_batch(it, b)
        its.append(it)
    which = rng.integers(0, len(depths), n)
    side = np.array([1 << d for d in depths])[which]
    xyz = (rng.random((n, 3)) * side[:, None]).astype(np.int32)
    want = its[0].get_many(handles[0][which], xyz)
    got = its[1].get_many(handles[1][which], xyz)
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_array_equal(got[0], want[0])
    if max(depths) > 1:
        assert (want[0].astype(bool) & (want[1] == 0)).any()
