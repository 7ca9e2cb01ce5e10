"""vx_interner_reset leaves the interner as created: whatever ran before it (builds, edits that left
tombstones, a table too full to be cleared key by key, a call that ran out of nodes or of table), the next
sequence of calls gives the BlockIds, counts and DAG of a fresh interner."""
import numpy as np
import pytest

from voxelis_gb300 import workloads as W
from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P4, VX_PATCH_P5, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree

PATCHES = VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5


def sequence(it, depth=4):
    rng = np.random.default_rng(3)
    trees = [VoxTree(depth) for _ in range(2)]
    log = []
    for t in trees:
        for p, v in zip(rng.integers(0, 1 << depth, (60, 3)), rng.integers(0, 4, 60)):
            t.set(it, p, int(v))
            log.append(t.get_root_id())
    s = it.stats()
    log += [s[k] for k in ("next_index", "free_count", "alive_nodes", "branch_patterns", "leaf_patterns",
                           "table_tombstones", "error_flags", "nodes_created")]
    return log, it.export_canonical(trees)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 16])
@pytest.mark.parametrize("before", ["build", "edits", "full table", "out of nodes", "table full"])
def test_reset_equals_a_fresh_interner(gpu_lib, bits, before):
    budget, log2 = 32 << 20, 0
    if before == "full table":
        log2 = 14
    if before == "out of nodes":
        budget = 300 * (79 + bits // 8 - 1)
    if before == "table full":
        log2 = 4
    it = VoxInterner(budget, bits, PATCHES, table_log2=log2, lib=gpu_lib)
    rng = np.random.default_rng(bits)
    trees = [VoxTree(5) for _ in range(4)]
    grids = rng.integers(0, 3, (4, 32, 32, 32)).astype(it.dtype)
    if before in ("build", "edits", "full table"):
        grids = W.dune_world_chunks(2, 2, depth=5, seed=5, dtype=it.dtype)
    try:
        it.build_dense(trees, grids)
        if before == "edits":
            for k in range(2):
                batches = []
                for t in trees:
                    b = t.create_batch(it)
                    b.set_many(rng.integers(0, 32, (200, 3)), rng.integers(0, 5, 200).astype(np.uint32))
                    batches.append(b)
                it.apply_batches(trees, batches)
            assert it.stats()["table_tombstones"] > 0
        assert before in ("build", "edits", "full table")
    except VoxelisError:
        assert before in ("out of nodes", "table full")
    it.lib.call("interner_reset", it.handle, handle=it.handle)
    for t in trees:
        assert t.get_root_id() == 0
    fresh = VoxInterner(budget, bits, PATCHES, table_log2=log2, lib=gpu_lib)
    for _ in trees:  # the same tree handles
        VoxTree(5)._bind(fresh)
    if before == "table full":  # 16 slots hold no such sequence: the fresh interner runs out as well
        for i in (it, fresh):
            s = i.stats()
            assert s["alive_nodes"] == 1 and s["error_flags"] == 0 and s["branch_patterns"] == 1
        return
    a, b = sequence(it, 3 if before == "out of nodes" else 4), sequence(fresh, 3 if before == "out of nodes" else 4)
    assert a[0] == b[0]
    for k in a[1]:
        np.testing.assert_array_equal(a[1][k], b[1][k])
