"""Batched applies at the record counts where the default changes between one launch and a launch per phase: the
oracle's DAG on both sides, with sets and then with clears (voxtree.rs:303-328, 724-1118)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P2, VX_PATCH_P3, VX_PATCH_P4, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree

PATCHES = VX_PATCH_P1 | VX_PATCH_P2 | VX_PATCH_P3 | VX_PATCH_P4 | VX_PATCH_P5


@pytest.mark.gpu
@pytest.mark.parametrize("records", [(1 << 17) - 1, 1 << 17, (1 << 19) - 1, 1 << 19])
def test_apply_around_the_line(oracle_lib, gpu_lib, records, depth=7):
    rng = np.random.default_rng(records)
    items = 3
    its, trees = [], []
    for lib in (oracle_lib, gpu_lib):
        its.append(VoxInterner(1 << 28, 8, PATCHES, lib=lib))
        trees.append([VoxTree(depth) for _ in range(items)])
    each = [records // 3, records // 3, records - 2 * (records // 3)]
    groups = [rng.permutation(1 << 18)[:n] for n in each]  # one voxel in each group, so as many records
    for step in range(2):
        work = []
        for g in groups:
            xyz = np.stack([g % 64, g // 64 % 64, g // 4096], 1) * 2 + rng.integers(0, 2, (len(g), 3))
            values = rng.integers(1, 4, len(g))
            if step:
                values[rng.random(len(g)) < 0.5] = 0
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
        assert its[0].stats()["alive_nodes"] == its[1].stats()["alive_nodes"]


@pytest.mark.gpu
@pytest.mark.parametrize("records", [(1 << 17) - 1, 1 << 17, (1 << 19) - 1, 1 << 19])
def test_deep_trees_around_the_line(oracle_lib, gpu_lib, records):
    test_apply_around_the_line(oracle_lib, gpu_lib, records, depth=8)
