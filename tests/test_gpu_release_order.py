"""Slots come back in the reference's order: after VoxTree::set, fill and clear (voxtree.rs:163-292) have
released whole subtrees (dec_ref_recursive, interner/mod.rs:419-534), the slots that later nodes take, and
so their raw BlockIds, are those of the one-by-one loop. Subtrees of more nodes than one step of the release
takes, children shared by many parents of a step, and parents with one child in several slots."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P3
from voxelis_gb300.api import VoxInterner, VoxTree


def both(oracle_lib, gpu_lib, bits, patches):
    return [VoxInterner(16 << 20, bits, patches, lib=lib) for lib in (oracle_lib, gpu_lib)]


@pytest.mark.gpu
@pytest.mark.parametrize("bits,depth,voxels,kinds,patches", [
    (8, 2, 12, 2, 0), (8, 4, 90, 1, 0), (8, 5, 300, 3, 0), (16, 5, 260, 4000, 0), (8, 5, 300, 40, VX_PATCH_P3),
])
def test_ids_after_release(oracle_lib, gpu_lib, bits, depth, voxels, kinds, patches):
    rng = np.random.default_rng(depth * 1000 + voxels)
    side = 1 << depth
    places = rng.integers(0, side, (3, voxels, 3))
    values = rng.integers(1, kinds + 1, (3, voxels))
    # one half of the first tree is a repeated 2x2x2 pattern, so subtrees are shared and repeat within nodes
    places[0, : voxels // 2] = [(x, y, z) for x, y, z in places[0, : voxels // 2] // 2 * 2]
    log = []
    for it in both(oracle_lib, gpu_lib, bits, patches):
        trees = [VoxTree(depth) for _ in range(3)]
        seen = []

        def note():
            seen.append([t.get_root_id() for t in trees] + [it.stats()[k] for k in ("next_index", "free_count")])

        for k in range(2):
            for p, v in zip(places[k], values[k]):
                trees[k].set(it, p, int(v))
            note()
        trees[0].clear(it)  # shares with tree 1 what stays
        note()
        for p, v in zip(places[2], values[2]):
            trees[2].set(it, p, int(v))
            if not seen or len(seen) < 40:
                note()
        trees[1].fill(it, 7)
        note()
        for p, v in zip(places[0][: voxels // 3], values[0]):
            trees[0].set(it, p, int(v))
        note()
        for p in places[2][: voxels // 2]:
            trees[2].set(it, p, 0)
        note()
        for t in trees:
            t.clear(it)
        note()
        log.append(seen)
    assert log[0] == log[1]
