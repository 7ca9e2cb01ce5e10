"""Batched applies of many shapes against the oracle: record counts around a tile of 32, around the largest
apply that runs as one cluster, and past it; one item with many records, many items with one, trees of all
depths in one call, items with a fill, with nothing, and with clears only (P4); as one launch and as a launch
per phase (voxtree.rs:303-328, 724-1118)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P2, VX_PATCH_P4, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree

PATCHES = VX_PATCH_P1 | VX_PATCH_P2 | VX_PATCH_P4 | VX_PATCH_P5


@pytest.mark.gpu
@pytest.mark.parametrize("single", [1, 0])
@pytest.mark.parametrize("bits,items,edits,depths", [
    (8, 1, 1, (2,)), (8, 1, 31, (5,)), (16, 1, 33, (9,)), (8, 1, 4000, (6,)), (16, 1, 9000, (6,)),
    (8, 40, 1, (2, 3, 4, 5, 6, 7)), (16, 300, 7, (2, 3, 4)), (8, 300, 20, (4, 5)), (8, 65, 64, (8, 3, 2)),
])
def test_apply_shapes(oracle_lib, gpu_lib, single, bits, items, edits, depths):
    rng = np.random.default_rng(1000 * items + edits)
    its, trees = [], []
    depth_of = [depths[k % len(depths)] for k in range(items)]
    for lib in (oracle_lib, gpu_lib):
        it = VoxInterner(256 << 20, bits, PATCHES, lib=lib)
        its.append(it)
        trees.append([VoxTree(d) for d in depth_of])
    its[1].lib.call("tune_set_launch", its[1].handle, single, handle=its[1].handle)
    for step in range(4):
        work = []
        for k in range(items):
            n = edits if step != 1 else max(1, edits // 2)
            xyz = rng.integers(0, 1 << depth_of[k], (n, 3)).astype(np.int32)
            values = rng.integers(1, 5, n).astype(np.uint32)
            if step >= 2:  # clears beside sets, then clears alone in most items
                values[rng.random(n) < (0.4 if step == 2 else 0.9)] = 0
            kind = (k + step) % 9
            work.append((xyz, values, kind))
        changed = []
        for it, ts in zip(its, trees):
            batches = []
            for t, (xyz, values, kind) in zip(ts, work):
                b = t.create_batch(it)
                if kind == 7 and step:
                    b.just_fill(int(1 + step))
                if not (kind == 8 and step == 1):  # that one leaves the batch empty or a bare fill
                    b.set_many(xyz, values)
                elif not (kind == 7 and step):
                    b.just_fill(2)
                batches.append(b)
            changed.append(it.apply_batches(ts, batches))
        np.testing.assert_array_equal(changed[0], changed[1])
        a, b = (it.export_canonical(ts) for it, ts in zip(its, trees))
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg="%s after step %d" % (key, step))
        assert its[0].stats()["alive_nodes"] == its[1].stats()["alive_nodes"]
        its[1].validate(trees[1])
