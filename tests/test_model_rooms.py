"""Model payloads larger than the room that the first call of serialize_model / deserialize_model offers: more bytes
than a megabyte, more chunks than 65536, and small ones beside them (world/voxmodel.rs:177-408)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P2
from voxelis_gb300.api import VoxInterner, VoxTree


def _round_trip(lib, budget, depth, trees_voxels):
    it = VoxInterner(budget, 8, VX_PATCH_P1 | VX_PATCH_P2, lib=lib)
    trees = [VoxTree(depth) for _ in trees_voxels]
    for t, (xyz, values) in zip(trees, trees_voxels):
        if len(xyz):
            b = t.create_batch(it)
            b.set_many(xyz, values)
            assert t.apply_batch(it, b)
    pos = np.arange(3 * len(trees), dtype=np.int32).reshape(-1, 3)
    blob = it.serialize_model(trees, pos)
    into = VoxInterner(budget, 8, VX_PATCH_P1 | VX_PATCH_P2, lib=lib)
    loaded, where = into.deserialize_model(blob, depth)
    np.testing.assert_array_equal(where, pos)
    assert len(loaded) == len(trees) and all(t.is_dirty() for t in loaded)
    for k in {0, len(trees) // 2, len(trees) - 1}:
        np.testing.assert_array_equal(loaded[k].to_vec(into), trees[k].to_vec(it))
    assert into.serialize_model(loaded, where) == blob
    return blob


@pytest.mark.gpu
@pytest.mark.parametrize("chunks,depth,voxels", [(1, 7, 300000), (66000, 2, 0), (3, 4, 50)])
def test_model_rooms(oracle_lib, gpu_lib, chunks, depth, voxels):
    rng = np.random.default_rng(chunks)
    none = (np.zeros((0, 3), np.int32), np.zeros(0, np.uint32))
    work = [none] * chunks
    for k in {0, chunks // 2, chunks - 1}:
        n = max(voxels, 3)
        work[k] = (rng.integers(0, 1 << depth, (n, 3)).astype(np.int32), rng.integers(1, 200, n).astype(np.uint32))
    blob = _round_trip(gpu_lib, 256 << 20, depth, work)
    if voxels == 300000:
        assert len(blob) > 1 << 20
    if chunks == 3:  # node indices, and so bytes, may differ from the oracle's; what they say may not
        other = VoxInterner(256 << 20, 8, VX_PATCH_P1 | VX_PATCH_P2, lib=oracle_lib)
        trees, _ = other.deserialize_model(blob, depth)
        for t, (xyz, values) in zip(trees, work):
            for p, v in {tuple(p): v for p, v in zip(xyz.tolist(), values.tolist())}.items():
                assert t.get(other, p) == v
