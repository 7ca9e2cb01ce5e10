"""Batches with sets and clears (P4) in interners with much, little and just enough room: the release of the set phase
waits for the clear pass where the free nodes allow it and goes before it where they do not; the oracle's DAG, counts
and live nodes either way, as one launch and as a launch per phase."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_E_OOM, VX_PATCH_P1, VX_PATCH_P4, VX_PATCH_P5, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree

PATCHES = VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5


def _steps(it, depth, edits, items, seed, each=None):
    """Rounds of batches with sets and clears; what the trees hold after each."""
    rng = np.random.default_rng(seed)
    trees = [VoxTree(depth) for _ in range(items)]
    out = []
    for step in range(5):
        batches = []
        for t in trees:
            xyz = rng.integers(0, 1 << depth, (edits, 3)).astype(np.int32)
            values = rng.integers(1, 4, edits).astype(np.uint32)
            if step:
                values[rng.random(edits) < 0.5] = 0
            b = t.create_batch(it)
            b.set_many(xyz, values)
            batches.append(b)
        changed = it.apply_batches(trees, batches)
        out.append((changed, it.export_canonical(trees), it.stats()["alive_nodes"]))
        if each:
            each(trees)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("single", [1, 0])
@pytest.mark.parametrize("depth,edits,items", [(4, 60, 3), (5, 1500, 2), (6, 9000, 1)])
def test_room_for_the_clear_pass(oracle_lib, gpu_lib, single, depth, edits, items):
    want = _steps(VoxInterner(64 << 20, 8, PATCHES, lib=oracle_lib), depth, edits, items, depth)
    peak = max(alive for _, _, alive in want)
    done = []
    for room in (20.0, 3.0, 2.4, 2.1, 1.9, 1.75, 1.6):  # times the largest number of live nodes
        it = VoxInterner(int(peak * room) * 79, 8, PATCHES, lib=gpu_lib)
        it.lib.call("tune_set_launch", it.handle, single, handle=it.handle)
        try:
            got = _steps(it, depth, edits, items, depth, it.validate)
        except VoxelisError as e:
            assert e.status == VX_E_OOM and room < 2  # the old and the new trees together do not fit
            continue
        done.append(room)
        for step, ((ca, da, na), (cb, db, nb)) in enumerate(zip(want, got)):
            np.testing.assert_array_equal(ca, cb)
            for key in da:
                np.testing.assert_array_equal(da[key], db[key], err_msg="%s, step %d, room %s" % (key, step, room))
            assert na == nb
    assert {20.0, 3.0, 2.4, 2.1} <= set(done)
