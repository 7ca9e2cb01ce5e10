"""The branch table under edits that come and go: the same keys are created and released again and again in a
small table, so most inserts meet tombstones, several lanes want the same one, and runs of deleted slots
wrap around the table's end. The DAG, refcounts and live counts stay the oracle's (set, clear and refill
batches on several trees at once; interner/mod.rs:566-625, 712-829), and tombstones do not pile up."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P4, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("bits,table_log2,single", [(8, 13, 1), (8, 13, 0), (16, 14, 1), (16, 0, 0)])
def test_keys_created_and_released_repeatedly(oracle_lib, gpu_lib, bits, table_log2, single):
    rng = np.random.default_rng(bits + table_log2)
    n, depth, rounds = 6, 4, 12
    patches = VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5
    xyz = [rng.integers(0, 16, (300, 3)).astype(np.int32) for _ in range(n)]
    values = [rng.integers(1, 6, 300).astype(np.uint32) for _ in range(n)]
    interners, trees = [], []
    for lib in (oracle_lib, gpu_lib):
        it = VoxInterner(8 << 20, bits, patches, table_log2=table_log2, lib=lib)
        interners.append(it)
        trees.append([VoxTree(depth) for _ in range(n)])
    gpu = interners[1]
    gpu.lib.call("tune_set_launch", gpu.handle, single, handle=gpu.handle)
    tombs = []
    for r in range(rounds):
        for it, ts in zip(interners, trees):
            batches = []
            for k, t in enumerate(ts):
                b = t.create_batch(it)
                v = values[k] if r % 2 == 0 else np.zeros_like(values[k])  # the carve takes every voxel away again
                b.set_many(xyz[k], v)
                batches.append(b)
            it.apply_batches(ts, batches)
        a, b = (it.export_canonical(ts) for it, ts in zip(interners, trees))
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg="%s, round %d" % (key, r))
        so, sg = (it.stats() for it in interners)
        assert so["alive_nodes"] == sg["alive_nodes"]
        gpu.validate(trees[1])
        tombs.append(sg["table_tombstones"])
    # the second half creates no key that the first half did not: it finds their tombstones again
    assert max(tombs[rounds // 2:]) <= 2 * max(tombs[:rounds // 2])
