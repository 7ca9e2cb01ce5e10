"""Several threads that read voxels of one interner at once, through host memory and in sizes that take every route of
the calls: each gets its own answers, errors among them."""
import threading

import numpy as np
import pytest

from voxelis_gb300 import workloads as W
from voxelis_gb300._abi import VX_E_OOB, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [8, 16])
def test_reads_from_several_threads(gpu_lib, bits):
    depth, n, side = 5, 12, 32
    it = VoxInterner(64 << 20, bits, lib=gpu_lib)
    trees = [VoxTree(depth) for _ in range(n)]
    grids = W.dune_world_chunks(4, 3, depth=depth, seed=2, dtype=it.dtype)
    it.build_dense(trees, grids)
    handles = np.array([t.tree for t in trees], np.uint32)
    failed = []

    def gets(seed, count):
        rng = np.random.default_rng(seed)
        which, xyz = rng.integers(0, n, count), rng.integers(0, side, (count, 3)).astype(np.int32)
        want = grids[which, xyz[:, 1], xyz[:, 2], xyz[:, 0]]
        found, values = it.get_many(handles[which], xyz)
        return np.array_equal(values, want) and np.array_equal(found, want != 0)

    def one(seed):
        k, (x, y, z) = seed % n, np.random.default_rng(seed).integers(0, side, 3)
        return (trees[k].get(it, (int(x), int(y), int(z))) or 0) == grids[k, y, z, x]

    def dense(seed):
        some = [(seed + k) % n for k in range(1 + seed % n)]
        return np.array_equal(it.to_vec_many([trees[k] for k in some]), grids[some])

    def outside(seed):
        try:
            it.get_many(handles[:1], np.array([[side, 0, 0]], np.int32))
        except VoxelisError as e:
            return e.status == VX_E_OOB
        return False

    def work(name, reads, first):
        for seed in range(first, first + 60):
            try:
                if not all(r(seed) for r in reads):
                    failed.append((name, seed))
            except Exception as e:  # noqa: BLE001
                failed.append((name, seed, e))

    jobs = [("small", [lambda s: gets(s, 1 + s % 4096)]), ("large", [lambda s: gets(s, (1 << 14) + 997 * (s % 60))]),
            ("one", [one, outside]), ("dense", [dense]), ("largest", [lambda s: s % 20 or gets(s, (1 << 20) + s)])]
    threads = [threading.Thread(target=work, args=(name, reads, 100 * k)) for k, (name, reads) in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    it.sync()
