"""Device-resident batched applies (vx_apply_groups_async) whose items are not what their records suggest: a fill
without the patches bit beside records, trees that fail the depth checks, groups outside their tree and records out of
order. An item's root is committed once, what is refused is left alone, and the other trees are as if it were not there
(the oracle's apply_batch of them, voxtree.rs:303-328, 724-1118), in one launch and in one a phase."""
import ctypes as C

import numpy as np
import pytest

from voxelis_gb300 import workloads as W
from voxelis_gb300._abi import VX_E_INVALID_ARG, VX_PATCH_P1, VX_PATCH_P3, VX_PATCH_P4, VX_PATCH_P5, VoxelisError
from voxelis_gb300.api import VoxInterner, VoxTree

pytestmark = pytest.mark.gpu
PATCHES = VX_PATCH_P1 | VX_PATCH_P3 | VX_PATCH_P4 | VX_PATCH_P5
FILL = 77


def records_of(rng, depth, n, clears=True):
    """n random voxel writes (a third of them clears) and their records."""
    xyz = rng.integers(0, 1 << depth, (n, 3)).astype(np.int32)
    v = rng.integers(1, 6, n).astype(np.uint32)
    if clears:
        v[::3] = 0
    return (xyz, v), W.edits_to_groups(depth, xyz, v)


def device_apply(it, handles, flags, recs, max_depth, item=None):
    """Queues the apply; returns its arrays, which live until the sync, the changed flags first."""
    import torch

    put = lambda a, t: torch.from_numpy(np.ascontiguousarray(a).view(t).copy()).cuda()  # noqa: E731
    item = np.concatenate([np.full(len(r[0]), i, np.uint32) for i, r in enumerate(recs)]) if item is None else item
    group, sets, clears, vals = (np.concatenate([r[j] for r in recs]) for j in range(4))
    n = len(handles)
    arrays = [torch.full((n,), 9, dtype=torch.uint8, device="cuda"), put(np.array(handles, np.uint32), np.int32),
              put(np.array(flags, np.uint8), np.uint8), put(np.full(n, FILL, np.uint32), np.int32),
              put(item.astype(np.uint32), np.int32), put(group, np.int32), put(sets, np.uint8), put(clears, np.uint8),
              put(vals.reshape(-1), np.int16)]
    torch.cuda.synchronize()
    p = [C.c_void_p(a.data_ptr()) for a in arrays]
    it._call("apply_groups_async", n, p[1], p[2], p[3], len(item), p[4], p[5], p[6], p[7], p[8], p[0], max_depth)
    return arrays


def pair(libs, depths, built, single):
    """The same trees in an interner of each library, the `built` ones with terrain in them."""
    out = []
    for lib in libs:
        it = VoxInterner(64 << 20, 8, PATCHES, lib=lib)
        trees = [VoxTree(d) for d in depths]
        for k, t in enumerate(trees):
            t._bind(it)
            if built and t.max_depth_value < 2:
                t.fill(it, 3)
            elif built:
                it.build_dense([t], W.dune_world_chunks(1, 1, depth=t.max_depth_value, seed=k))
        out.append((it, trees))
    out[1][0]._call("tune_set_launch", single)
    return out


def same_state(a, b, ta, tb, leaf_refs=0):
    """leaf_refs: references that the fill's leaf has in a beyond b's."""
    ca, cb = a.export_canonical(ta), b.export_canonical(tb)
    fill = (ca["kind"] == 1) & (ca["value"] == FILL)  # the leaf
    refs = ca["refcount"].astype(np.int64) - np.where(fill, leaf_refs, 0)
    for k in ca:
        np.testing.assert_array_equal(refs if k == "refcount" else ca[k], cb[k], err_msg=k)


@pytest.mark.parametrize("single", [1, 0])
@pytest.mark.parametrize("writes", [20, 20000])
@pytest.mark.parametrize("built", [False, True])
def test_fill_without_the_patches_bit(oracle_lib, gpu_lib, single, writes, built):
    depth, n = 5, 3
    (oi, ot), (gi, gt) = pair((oracle_lib, gpu_lib), (depth,) * n, built, single)
    rng = np.random.default_rng(writes)
    work = [records_of(rng, depth, writes, clears=k != 1) for k in range(n)]
    batches = []
    for t, (edits, _) in zip(ot, work):
        b = t.create_batch(oi)
        b.fill(oi, FILL)
        b.set_many(*edits)
        batches.append(b)
    want = oi.apply_batches(ot, batches)
    arrays = device_apply(gi, [t.tree for t in gt], [1] * n, [w[1] for w in work], depth)
    gi.sync()
    np.testing.assert_array_equal(arrays[0].cpu().numpy().astype(bool), want)
    # the oracle's batches have patches: a reference for the fill each (voxtree.rs:742-758)
    same_state(oi, gi, ot, gt, leaf_refs=n)
    assert oi.stats()["alive_nodes"] == gi.stats()["alive_nodes"]


@pytest.mark.parametrize("single", [1, 0])
def test_fill_whose_records_change_nothing(oracle_lib, gpu_lib, single):
    depth = 4
    (oi, ot), (gi, gt) = pair((oracle_lib, gpu_lib), (depth, depth), True, single)
    oi.apply_batches(ot, [_filled(t, oi) for t in ot])
    r = (np.arange(5, dtype=np.uint32), np.full(5, 3, np.uint8), np.zeros(5, np.uint8), np.full((5, 8), FILL, np.uint16))
    none = tuple(x[:0] for x in r)
    arrays = device_apply(gi, [t.tree for t in gt], [1, 1], [r, none], depth)
    gi.sync()
    assert arrays[0].cpu().tolist() == [1, 1]
    np.testing.assert_array_equal(gi.to_vec_many(gt), oi.to_vec_many(ot))
    assert oi.stats()["alive_nodes"] == gi.stats()["alive_nodes"]


def _filled(tree, it):
    b = tree.create_batch(it)
    b.fill(it, FILL)
    return b


@pytest.mark.parametrize("single", [1, 0])
@pytest.mark.parametrize("writes", [100, 20000])
@pytest.mark.parametrize("refused", ["unknown", "destroyed", "too deep", "out of order", "too shallow"])
def test_refused_trees_leave_the_others_alone(oracle_lib, gpu_lib, refused, writes, single):
    depths = {"too deep": (6, 5, 5, 5), "out of order": (5, 4, 5, 5), "too shallow": (5, 5, 5, 1)}.get(refused, (5, 5, 5, 5))
    bad = {"too deep": 0, "too shallow": 3}.get(refused, 2)
    take = [0, 1, 2] if refused == "out of order" else [0, 1, 2, 3]  # (a tree after one out of order is not promised)
    (oi, ot), (gi, gt) = pair((oracle_lib, gpu_lib), depths, True, single)
    rng = np.random.default_rng(writes)
    work = [records_of(rng, max(2, d), writes) for d in depths]
    handles = [t.tree for t in gt]
    if refused == "unknown":
        handles[bad] = 1 << 30
    if refused == "destroyed":
        for it, trees in ((oi, ot), (gi, gt)):
            trees[bad].clear(it)
        gi._call("tree_destroy", handles[bad])
    before = None if refused in ("unknown", "destroyed") else gi.to_vec_many([gt[bad]])
    good = [k for k in take if k != bad]
    batches = []
    for k in good:
        b = ot[k].create_batch(oi)
        b.set_many(*work[k][0])
        batches.append(b)
    want = oi.apply_batches([ot[k] for k in good], batches)
    arrays = device_apply(gi, [handles[k] for k in take], [2] * len(take), [work[k][1] for k in take], 5)
    with pytest.raises(VoxelisError) as e:
        gi.sync()
    assert e.value.status == VX_E_INVALID_ARG
    changed = arrays[0].cpu().numpy()
    np.testing.assert_array_equal(changed[[take.index(k) for k in good]].astype(bool), want)
    assert changed[take.index(bad)] == 0
    if before is not None:
        np.testing.assert_array_equal(gi.to_vec_many([gt[bad]]), before)
    rest = [k for k in range(4) if k != bad or refused != "destroyed"]
    gi.validate([gt[k] for k in rest])
    same_state(oi, gi, [ot[k] for k in rest], [gt[k] for k in rest])
    assert oi.stats()["alive_nodes"] == gi.stats()["alive_nodes"]


@pytest.mark.parametrize("single", [1, 0])
@pytest.mark.parametrize("form", ["outside", "out of order"])
def test_records_that_name_no_place_once(gpu_lib, form, single):
    (_, _), (gi, gt) = pair((gpu_lib, gpu_lib), (5, 5, 4), True, single)
    before = gi.to_vec_many(gt[:2])
    rng = np.random.default_rng(1)
    recs = [records_of(rng, 5, 3000, False)[1], records_of(rng, 4, 300, False)[1]]
    item = None
    if form == "outside":  # all of the second tree's groups, and one of the first one's
        recs[0][0][-1] |= 1 << 12
        recs[1][0][:] |= 1 << 20
    else:
        item = np.concatenate([np.arange(len(recs[0][0])) % 2, np.full(len(recs[1][0]), 1)])
        recs[0][0][:] = rng.permutation(recs[0][0])
    arrays = device_apply(gi, [gt[0].tree, gt[2].tree], [2, 2], recs, 5, item)
    with pytest.raises(VoxelisError) as e:
        gi.sync()
    assert e.value.status == VX_E_INVALID_ARG
    np.testing.assert_array_equal(gi.to_vec_many([gt[1]])[0], before[1])
    if form == "outside":
        assert arrays[0].cpu().tolist() == [1, 0]
        gi.validate(gt)
        got = gi.to_vec_many([gt[0]])[0]
        want = before[0].copy()
        for g, m, v in zip(recs[0][0][:-1], recs[0][1][:-1], recs[0][3][:-1]):
            for k in range(8):
                if m >> k & 1:
                    x, y, z = (sum(((int(g) << 3 | k) >> (3 * b + a) & 1) << b for b in range(5)) for a in range(3))
                    want[y, z, x] = v[k]
        np.testing.assert_array_equal(got, want)
