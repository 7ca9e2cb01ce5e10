"""Branch tables smaller than, as large as and larger than the four slots that a probe reads: every slot is used,
and the key that no slot is left for is refused (batched applies and batched single-voxel calls)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_E_TABLE_FULL, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("many", [0, 1])
@pytest.mark.parametrize("table_log2,depth", [(1, 2), (2, 4), (3, 4), (3, 5), (4, 5)])
def test_every_slot_is_used_and_no_more(gpu_lib, table_log2, depth, many):
    rng = np.random.default_rng(table_log2 * 8 + depth)
    slots = 1 << table_log2
    for trial in range(8):  # other hashes, so other first slots and wraps
        it = VoxInterner(1 << 20, 8, 0, table_log2=table_log2, lib=gpu_lib)
        used, value = 0, 1
        while True:  # a voxel alone in its tree makes one branch a level
            tree, p = VoxTree(depth), [int(x) for x in rng.integers(0, 1 << depth, 3)]
            fits = used + depth <= slots

            def edit():
                if many:
                    return bool(it.set_many([tree], [p], [value])[0])
                b = tree.create_batch(it)
                b.just_set(p, value)
                return tree.apply_batch(it, b)

            if not fits:
                with pytest.raises(VoxelisError) as e:
                    edit()
                    it.sync()
                assert e.value.status == VX_E_TABLE_FULL
                break
            assert edit()
            assert tree.get(it, p) == value
            used, value = used + depth, value + 1
            assert it.stats()["alive_nodes"] >= used
        it.close()
