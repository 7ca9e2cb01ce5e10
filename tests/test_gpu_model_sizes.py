"""Model payloads of many sizes (VoxModel::serialize / deserialize, world/voxmodel.rs:177-408): from a few
records to several parse groups of 2 KB, sections that end anywhere in a group, and payloads past 2 MB,
whose segments are longer. The oracle writes each payload; the GPU library loads it and must hold the
oracle's DAG and write the same bytes again."""
import numpy as np
import pytest

from voxelis_gb300.api import VoxInterner, VoxTree


def model(lib, bits, n, depth, seed, kinds):
    """n chunks of noise with `kinds` values; few chunks share nodes, so the payload grows with n."""
    rng = np.random.default_rng(seed)
    it = VoxInterner(512 << 20, bits, lib=lib)
    trees = [VoxTree(depth) for _ in range(n)]
    side = 1 << depth
    grids = rng.integers(0, kinds, (n, side, side, side)).astype(it.dtype)
    it.build_dense(trees, grids)
    return it, trees, rng.integers(-1000, 1000, (n, 3)).astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,n,depth,kinds", [
    (8, 1, 2, 2), (16, 1, 3, 300), (8, 3, 3, 5), (16, 7, 3, 3), (8, 20, 3, 200), (16, 33, 4, 2000), (8, 97, 2, 4),
    (16, 130, 5, 4000),
])
def test_payload_sizes(oracle_lib, gpu_lib, bits, n, depth, kinds):
    io, to, pos = model(oracle_lib, bits, n, depth, 31 * n + depth, kinds)
    payload = io.serialize_model(to, pos)
    assert n < 130 or len(payload) > 1 << 21
    got = []
    for lib in (oracle_lib, gpu_lib):
        it = VoxInterner(512 << 20, bits, lib=lib)
        trees, positions = it.deserialize_model(payload, depth)
        np.testing.assert_array_equal(positions, pos)
        got.append(it.export_canonical(trees))
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
    assert it.serialize_model(trees, pos) == payload  # a loaded model's slots are its record ids
