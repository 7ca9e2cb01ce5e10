"""Sphere brushes staged by the device are those that the host stages: items, their trees and spheres, and every record,
for all chunk depths it takes, spheres over chunk edges, past the world's edges and larger than a chunk, single
voxels, carves; what it does not take is refused with nothing written (batch.rs:145-172)."""
import ctypes as C

import numpy as np
import pytest

from voxelis_gb300._abi import VX_E_BUFFER, VX_E_INVALID_ARG, VX_E_UNSUPPORTED, VX_PATCH_P2
from voxelis_gb300.serve import World

CAP = 1 << 16


def _host(lib, w, cen, rad, val, cap_recs):
    out = [np.zeros(CAP, np.uint32), np.zeros(cap_recs, np.uint32), np.zeros(cap_recs, np.uint32), np.zeros(cap_recs, np.uint8),
           np.zeros(cap_recs, np.uint8), np.zeros((cap_recs, 8), np.uint16)]
    ni, nr = C.c_uint64(), C.c_uint64()
    f = lib.lib.vx_stage_spheres
    f.restype = C.c_int
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    st = f(w.depth, w.nx, w.ny, w.nz, len(rad), P(cen), P(rad), P(val), C.c_uint64(CAP), P(out[0]), C.c_uint64(cap_recs),
           *[P(a) for a in out[1:]], C.byref(ni), C.byref(nr))
    return st, ni.value, nr.value, out


def _device(lib, w, cen, rad, val, cap_recs):
    import torch

    new = lambda n, dt: torch.zeros(n, dtype=dt, device="cuda")  # noqa: E731
    plan = torch.zeros(8 * CAP, dtype=torch.int32).pin_memory()
    items = [new(8 * CAP, torch.int32)] + [new(CAP, torch.int32) for _ in range(3)]
    recs = [new(cap_recs, torch.int32), new(cap_recs, torch.int32), new(cap_recs, torch.uint8), new(cap_recs, torch.uint8),
            new(cap_recs * 8, torch.int16)]
    ni, nr = C.c_uint64(), C.c_uint64()
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    st = lib.status("stage_spheres_async", w.h, C.byref(w.wdesc), len(rad), cen.ctypes.data, rad.ctypes.data, val.ctypes.data,
                    CAP, P(plan), *[P(t) for t in items], cap_recs, *[P(t) for t in recs], C.byref(ni), C.byref(nr))
    w.call("interner_sync")
    return st, ni.value, nr.value, [t.cpu().numpy() for t in items[1:] + recs]


def _spheres(rng, w, count, r_max):
    """Spheres whose boxes touch disjoint chunks; some centres are outside of the world."""
    side, size = w.side, [k * w.side for k in (w.nx, w.ny, w.nz)]
    used, out = set(), []
    for _ in range(200):
        c = [int(rng.integers(-side // 2, s + side // 2 + 1)) for s in size]
        r = int(rng.integers(0, r_max + 1))
        box = [range(max(0, c[k] - r) // side, min(size[k] - 1, c[k] + r) // side + 1) for k in range(3)]
        touched = {(x, y, z) for x in box[0] for y in box[1] for z in box[2]}
        if touched & used:
            continue
        used |= touched
        out.append((c, r, int(rng.integers(0, 3)) * 100))
        if len(out) == count:
            break
    return (np.array([c for c, _, _ in out], np.int32), np.array([r for _, r, _ in out], np.int32),
            np.array([v for _, _, v in out], np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("depth,shape,r_max", [(1, (9, 4, 5), 1), (2, (7, 3, 5), 3), (3, (5, 4, 6), 9), (4, (4, 3, 5), 6),
                                              (5, (4, 2, 4), 12), (6, (6, 2, 6), 12), (6, (2, 2, 2), 100), (7, (3, 2, 2), 40), (8, (2, 1, 1), 30)])
def test_records_are_the_hosts(gpu_lib, depth, shape, r_max):
    rng = np.random.default_rng(100 * depth + r_max)
    w = World(*shape, depth, budget=64 << 20, patches=VX_PATCH_P2, lib=gpu_lib)
    caps = 1 << 18 if depth < 6 else 1 << 20
    for count in (1, 1, 3, 20):
        cen, rad, val = _spheres(rng, w, count, r_max)
        sh, ih, rh, host = _host(gpu_lib, w, cen, rad, val, caps)
        sd, idv, rd, dev = _device(gpu_lib, w, cen, rad, val, caps)
        assert (sh, ih, rh) == (sd, idv, rd) and sh == 0
        trees, chunks, ranks, recs = dev[0], dev[1], dev[2], dev[3:]
        np.testing.assert_array_equal(chunks[:ih].view(np.uint32), host[0][:ih])
        np.testing.assert_array_equal(trees[:ih].view(np.uint32), w.trees[host[0][:ih]])
        for a, b in zip(recs, host[1:]):
            np.testing.assert_array_equal(a.view(b.dtype).reshape(b.shape)[:rh], b[:rh])
            assert not a.view(b.dtype).reshape(b.shape)[rh:].any()  # nothing behind the records
        for k in range(ih):  # the sphere of an item touches its chunk
            one = slice(int(ranks[k]), int(ranks[k]) + 1)
            _, n, _, only = _host(gpu_lib, w, cen[one], rad[one], val[one], caps)
            assert host[0][k] in only[0][:n]
    w.close()


@pytest.mark.gpu
def test_what_it_does_not_take(gpu_lib):
    w = World(3, 2, 2, 5, budget=64 << 20, lib=gpu_lib)
    i32, u32 = lambda *a: np.array(a, np.int32), lambda *a: np.array(a, np.uint32)  # noqa: E731
    for cen, rad, val, caps, want in (
            (i32((9, 9, 9), (40, 9, 9)), i32(3, 20), u32(1, 2), 4096, VX_E_UNSUPPORTED),  # both touch chunk 0
            (i32((9, 9, 9), (9, 9, 9)), i32(0, 0), u32(1, 0), 4096, VX_E_UNSUPPORTED),
            (i32((9, 9, 9)), i32(-1), u32(1), 4096, VX_E_INVALID_ARG),
            (i32((9, 9, 9)), i32(1), u32(1 << 16), 4096, VX_E_INVALID_ARG),
            (i32((32, 32, 32)), i32(12), u32(1), 64, VX_E_BUFFER),
            (i32((-50, 9, 9)), i32(5), u32(1), 64, 0)):
        cen = cen.reshape(-1, 3)
        st, ni, nr, dev = _device(gpu_lib, w, cen, rad, val, caps)
        assert st == want
        assert not any(a.any() for a in dev)
        if want in (VX_E_BUFFER, 0):
            assert (want, ni, nr) == _host(gpu_lib, w, cen, rad, val, caps)[:3]
    w.close()
    w = World(1, 1, 1, 9, budget=64 << 20, patches=VX_PATCH_P2, lib=gpu_lib)
    assert _device(gpu_lib, w, i32((9, 9, 9)).reshape(-1, 3), i32(3), u32(1), 4096)[0] == VX_E_UNSUPPORTED
    w.close()
