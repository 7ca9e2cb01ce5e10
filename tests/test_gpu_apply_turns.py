"""Batched applies whose CTAs share the bottom groups out in turn (four tiles of records a warp and more), reached at
small sizes by launching few and small CTAs: around the line, with ranges that do not divide evenly among the
warps, with clears (P4), against the oracle (voxtree.rs:303-328, 724-1118)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P4, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("threads,bits,items,groups", [
    (32, 8, 4, 4864), (32, 16, 5, 4100), (32, 8, 3, 9001), (96, 16, 9, 8192), (64, 8, 7, 6007),
])
def test_bottom_groups_in_turn(oracle_lib, gpu_lib, threads, bits, items, groups):
    rng = np.random.default_rng(threads + groups)
    depth = 6  # 32768 groups a tree
    its, trees = [], []
    for lib in (oracle_lib, gpu_lib):
        its.append(VoxInterner(256 << 20, bits, VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5, lib=lib))
        trees.append([VoxTree(depth) for _ in range(items)])
    its[1].lib.call("tune_set", its[1].handle, threads, 1, handle=its[1].handle)
    for step in range(3):
        work = []
        for _ in range(items):
            g = rng.permutation(32768)[:groups]  # one voxel in each group, so as many records
            xyz = np.stack([g % 32, g // 32 % 32, g // 1024], 1) * 2 + rng.integers(0, 2, (groups, 3))
            values = rng.integers(1, 4, groups)
            if step == 2:
                values[rng.random(groups) < 0.5] = 0
            work.append((xyz.astype(np.int32), values.astype(np.uint32)))
        changed = []
        for it, ts in zip(its, trees):
            batches = [t.create_batch(it) for t in ts]
            for b, (xyz, values) in zip(batches, work):
                b.set_many(xyz, values)
            changed.append(it.apply_batches(ts, batches))
        np.testing.assert_array_equal(changed[0], changed[1])
        a, b = (it.export_canonical(ts) for it, ts in zip(its, trees))
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg="%s after step %d" % (key, step))
        its[1].validate(trees[1])
