"""Clearing trees of thousands of nodes: levels wider than one step of the release, queues longer than what it keeps in
shared memory, and both widths of its steps in turn leave the free list in the reference's order
(dec_ref_recursive, interner/mod.rs:419-534)."""
import numpy as np
import pytest

from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("bits,depth,voxels,kinds", [(8, 5, 33, 3), (8, 5, 700, 2), (8, 6, 5000, 200), (16, 6, 2500, 60000)])
def test_order_after_clear(oracle_lib, gpu_lib, bits, depth, voxels, kinds):
    rng = np.random.default_rng(voxels)
    places = rng.integers(0, 1 << depth, (voxels, 3))
    values = rng.integers(1, kinds + 1, voxels)
    log = []
    for lib in (oracle_lib, gpu_lib):
        it = VoxInterner(32 << 20, bits, 0, lib=lib)
        a, b = VoxTree(depth), VoxTree(depth)
        seen = []
        for k, (p, v) in enumerate(zip(places, values)):
            a.set(it, p, int(v))
            if k % 3 == 0:
                b.set(it, p, int(v))  # shares nodes with a
        a.clear(it)
        seen.append([it.stats()[k] for k in ("next_index", "free_count")])
        for p, v in zip(places[:200], values):
            b.set(it, p[::-1], int(v))  # takes slots from the free list
            seen.append(b.get_root_id())
        b.fill(it, 5)
        a.set(it, places[0], 9)
        seen += [a.get_root_id(), b.get_root_id()]
        log.append(seen)
    assert log[0] == log[1]
