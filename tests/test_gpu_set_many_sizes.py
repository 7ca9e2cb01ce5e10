"""vx_trees_set_many on both sides of the size up to which its arguments pass through pinned memory: the oracle's
one-by-one calls (VoxTree::set, voxtree.rs:163-260), and no host memory kept for large calls."""
import numpy as np
import pytest

from voxelis_gb300._abi import VX_PATCH_P3, VX_PATCH_P5
from voxelis_gb300.api import VoxInterner, VoxTree


@pytest.mark.gpu
@pytest.mark.parametrize("calls", [(1 << 16) - 1, 1 << 16, (1 << 16) + 1])
def test_calls_around_the_line(oracle_lib, gpu_lib, calls):
    depth, n = 3, 500
    rng = np.random.default_rng(calls)
    which, xyz = rng.integers(0, n, calls), rng.integers(0, 1 << depth, (calls, 3)).astype(np.int32)
    values = rng.integers(0, 4, calls).astype(np.uint32)
    oi, gi = (VoxInterner(64 << 20, 8, VX_PATCH_P3 | VX_PATCH_P5, lib=lib) for lib in (oracle_lib, gpu_lib))
    ot, gt = ([VoxTree(depth) for _ in range(n)] for _ in range(2))
    want = np.array([ot[k].set(oi, p, int(v)) for k, p, v in zip(which, xyz.tolist(), values)])
    for t in ot + gt:
        t._bind(oi if t in ot else gi)
    got = gi.set_many([gt[k] for k in which], xyz, values)
    np.testing.assert_array_equal(got, want)
    a, b = oi.export_canonical(ot), gi.export_canonical(gt)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


def _resident_bytes():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) << 10 for line in f if line.startswith("VmRSS"))


@pytest.mark.gpu
def test_large_calls_keep_no_host_memory(gpu_lib):
    n = 256
    it = VoxInterner(64 << 20, lib=gpu_lib)
    trees = [VoxTree(2) for _ in range(n)]
    handles = np.array([t._bind(it) for t in trees], np.uint32)

    def calls(m):  # the same voxel of a tree again and again
        which = np.arange(m) % n
        args = handles[which], np.zeros((m, 3), np.int32), np.full(m, 3, np.uint32)
        changed = np.zeros(m, np.uint8)
        it._call("trees_set_many", m, *(a.ctypes.data for a in args), changed.ctypes.data)
        return changed

    assert calls(1 << 18).sum() == n
    before = _resident_bytes()
    m = 1 << 22
    assert calls(m).sum() == 0
    assert _resident_bytes() - before < 25 * m // 2
