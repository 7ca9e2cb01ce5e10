"""vx_trees_set_many on trees with many calls (their octants side by side) leaves what the oracle's one-by-one calls leave:
results, DAG, counts, live nodes. Roots that collapse into a leaf and split again, become EMPTY and come back, keep a
leaf's type bit after a set has split it, and collapse into a branch when 8 octants are equal under such bits
(voxtree.rs:163-260, 373-705)."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P1, VX_PATCH_P2, VX_PATCH_P4, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree

ALL = VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5


def _same(its, trees, step):
    a, b = (it.export_canonical(ts) for it, ts in zip(its, trees))
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg="%s after step %s" % (key, step))
    assert its[0].stats()["alive_nodes"] == its[1].stats()["alive_nodes"]
    its[1].validate(trees[1])


def _run(its, trees, which, xyz, values, step):
    one = [bool(trees[0][t].set(its[0], p, int(v))) for t, p, v in zip(which, xyz.tolist(), values)]
    many = its[1].set_many([trees[1][t] for t in which], xyz, values)
    np.testing.assert_array_equal(np.array(one), many, err_msg=str(step))
    _same(its, trees, step)


def _pair(oracle_lib, gpu_lib, bits, patches, depths):
    its = [VoxInterner(64 << 20, bits, patches, lib=lib) for lib in (oracle_lib, gpu_lib)]
    return its, [[VoxTree(d) for d in depths] for _ in its]


@pytest.mark.gpu
@pytest.mark.parametrize("bits,patches,depths,calls,kinds", [
    (8, 0, (2,), 4, 1), (8, 0, (2, 2, 2), 300, 1), (8, ALL, (3, 2, 5), 31, 2), (16, ALL | VX_PATCH_P2, (5, 7, 1, 4), 640, 3),
    (8, 0, (5,), 1000, 5), (16, 0, (4, 4, 3, 6, 2, 1, 5), 29, 60000),
])
def test_calls_in_order(oracle_lib, gpu_lib, bits, patches, depths, calls, kinds):
    rng = np.random.default_rng(calls + kinds)
    its, trees = _pair(oracle_lib, gpu_lib, bits, patches, depths)
    for step in range(5):
        which = rng.integers(0, len(depths), calls)
        xyz = np.array([rng.integers(0, 1 << depths[t], 3) for t in which], np.int32)
        values = rng.integers(1, kinds + 1, calls).astype(np.uint32)
        values[rng.random(calls) < (0.0, 0.3, 0.6, 0.0, 1.0)[step]] = 0
        _run(its, trees, which, xyz, values, step)
        if step == 1:  # the next calls meet a root that is a leaf
            for it, ts in zip(its, trees):
                ts[0].fill(it, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [2, 3])
def test_roots_collapse_and_split(oracle_lib, gpu_lib, depth):
    its, trees = _pair(oracle_lib, gpu_lib, 8, 0, (depth, depth))
    rng = np.random.default_rng(depth)
    side = 1 << depth
    cells = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    runs = []
    for value in (3, 0, 4, 3, 0):  # all of one value in any order, then split, then emptied
        runs += [(rng.permutation(cells), value), (cells[rng.integers(0, len(cells), 5)], 7)]
    xyz = np.concatenate([c for c, _ in runs]).astype(np.int32)
    values = np.concatenate([np.full(len(c), v) for c, v in runs]).astype(np.uint32)
    for cut in (len(xyz), 2 * len(cells) + 7, 40):  # whole, and from other states of the root
        _run(its, trees, np.arange(cut) % 2 if cut == 40 else np.zeros(cut, int), xyz[:cut], values[:cut], cut)


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [2, 4])
def test_eight_equal_octants(oracle_lib, gpu_lib, depth):
    its, trees = _pair(oracle_lib, gpu_lib, 8, 0, (depth,))
    for it, ts in zip(its, trees):
        ts[0].fill(it, 5)
    half = 1 << (depth - 1)
    corner = [[half * (o & 1), half * (o >> 1 & 1), half * (o >> 2)] for o in range(8)]
    xyz, values = [corner[o] for o in (1, 2, 3, 4, 5, 6, 7, 0)], [9] * 8
    xyz += [corner[0], corner[0]]  # back to a leaf, whose type bit then stays when it is split again
    values += [5, 9]
    xyz, values = np.array(xyz, np.int32), np.array(values, np.uint32)
    _run(its, trees, np.zeros(len(xyz), int), xyz, values, "equal octants")
    more = np.array([[0, 0, 0], [1, 1, 1], [half, 0, 0], [0, half, 1]], np.int32)
    _run(its, trees, np.zeros(4, int), more, np.array([2, 0, 3, 9], np.uint32), "after them")
