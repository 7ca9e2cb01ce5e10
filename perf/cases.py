"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public entry points: the Python classes of voxelis_gb300.api and
voxelis_gb300.serve, or the C ABI (VoxInterner.lib.call) for the calls that take device memory. Worlds
are dune terrain (u8 / u16 chunks) or 3D-noise caves (one deep tree), generated on the GPU from the seed.
A pass leaves a state that the next pass finds as it was, so it can be repeated: a build starts from a
reset interner, an edit is followed by the edit that takes it back.

listed()             the cases, smallest first within each kind
draw(rng)            one more case of the same ranges
prepare(case, seed)  the inputs and the interner a program has in hand before the call
run(state)           one pass; returns what it computes
work(case)           the bytes a pass cannot do without
exact(case, seed)    the outputs that follow from the inputs without this library
"""
import ctypes as C
import math

import numpy as np
import torch

from voxelis_gb300 import workloads as W
from voxelis_gb300._abi import (VX_MEM_DEVICE, VX_MEM_HOST, VX_PATCH_P1, VX_PATCH_P2, VX_PATCH_P3, VX_PATCH_P4,
                                VX_PATCH_P5)
from voxelis_gb300.api import VoxInterner, VoxTree
from voxelis_gb300.serve import EDIT, GET, Server, World, sphere_chunks

MAX_MATERIALS = 8     # materials a mesher asks the occupancy masks for
PLANES = 3 * 64 * 64  # words of a 64^3 builder's three mask planes
POINTS_PER_GET = 65536
FILE_PER_CHUNK = 4096  # room in a program's file buffer for each chunk of a model
EDITING = VX_PATCH_P1 | VX_PATCH_P4 | VX_PATCH_P5  # the patches of programs that edit worlds with carves


def listed():
    return [
        # a player places and takes away one block: the smallest call, pure latency
        {"name": "point_edit", "kind": "points", "bits": 8, "depth": 5, "chunks": 1, "edits": 1},
        # a simulation tick's scattered single-voxel edits over the loaded chunks, in one call
        {"name": "point_edits_4096", "kind": "points", "bits": 8, "depth": 5, "chunks": 64, "edits": 4096},
        # an editor's session on one chunk through the Python classes: load it dense, apply a host Batch,
        # probe a few voxels, read the chunk back
        {"name": "chunk_session", "kind": "session", "bits": 8, "depth": 5, "chunks": 1, "edits": 1000},
        # random reads over a loaded world of shallow chunks (physics, line of sight)
        {"name": "gets_chunks", "kind": "gets", "bits": 8, "depth": 5, "chunks": 4096, "queries": 1 << 22},
        # random reads of one deep tree
        {"name": "gets_caves", "kind": "gets", "bits": 8, "depth": 9, "chunks": 1, "queries": 1 << 24},
        # a whole world built from dense chunks on the device, then read back dense (the headline shape)
        {"name": "build_4096", "kind": "build", "bits": 8, "depth": 5, "chunks": 4096, "host": False},
        # a voxeliser's import: larger 16-bit chunks, grids in pinned host memory
        {"name": "build_host_u16", "kind": "build", "bits": 16, "depth": 6, "chunks": 256, "host": True},
        # a batch of edits of uneven density over chunks of three sizes, as device records, and its undo
        {"name": "uneven_edits", "kind": "uneven", "bits": 16, "depth": 7, "chunks": 96, "density": 0.1},
        # a server's backlog of sphere brushes and reads over a resident world
        {"name": "serve_backlog", "kind": "serve", "depth": 6, "nx": 16, "ny": 2, "nz": 16, "edits": 44, "gets": 20},
        # random sets and clears over one deep tree, and their undo
        {"name": "edit_caves", "kind": "deep", "bits": 8, "depth": 9, "edits": 1 << 18},
        # the masks a greedy mesher needs for every 64^3 builder of a world
        {"name": "masks_4096", "kind": "masks", "depth": 5, "chunks": 4096},
        # a model file's payload loaded into an empty interner and written again
        {"name": "model_round_trip", "kind": "model", "bits": 8, "depth": 5, "chunks": 1024},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["points", "session", "gets", "build", "uneven", "serve", "deep", "masks", "model"])
    bits = rng.choice([8, 16])
    if kind == "points":
        chunks = _log_int(rng, 1, 64)
        return {"kind": kind, "bits": bits, "depth": rng.randint(4, 6), "chunks": chunks,
                "edits": _log_int(rng, chunks, 4096)}
    if kind == "session":
        return {"kind": kind, "bits": bits, "depth": rng.randint(4, 6), "chunks": _log_int(rng, 1, 16),
                "edits": _log_int(rng, 10, 4000)}
    if kind == "gets":
        if rng.random() < 0.4:
            return {"kind": kind, "bits": bits, "depth": rng.randint(7, 9), "chunks": 1,
                    "queries": _log_int(rng, 1000, 1 << 24)}
        depth = rng.randint(3, 6)
        return {"kind": kind, "bits": bits, "depth": depth, "chunks": _log_int(rng, 16, 4096 >> max(0, 3 * (depth - 5))),
                "queries": _log_int(rng, 1000, 1 << 22)}
    if kind == "build":
        depth = rng.randint(3, 8)
        most = ((1 << 27) * 8 // bits) >> (3 * depth)
        return {"kind": kind, "bits": bits, "depth": depth, "chunks": _log_int(rng, 1, max(1, min(4096, most))),
                "host": rng.random() < 0.4}
    if kind == "uneven":
        return {"kind": kind, "bits": bits, "depth": rng.randint(5, 7), "chunks": _log_int(rng, 4, 96),
                "density": round(math.exp(rng.uniform(math.log(0.003), math.log(0.1))), 5)}
    if kind == "serve":
        return {"kind": kind, "depth": 6, "nx": rng.randint(4, 16), "ny": rng.randint(1, 2), "nz": rng.randint(4, 16),
                "edits": 2 * rng.randint(2, 22), "gets": rng.randint(1, 20)}
    if kind == "deep":
        depth = rng.randint(7, 9)
        return {"kind": kind, "bits": bits, "depth": depth, "edits": _log_int(rng, 500, 1 << (3 * depth - 9))}
    if kind == "masks":
        depth = rng.randint(4, 6)
        return {"kind": kind, "depth": depth, "chunks": _log_int(rng, 3, 4096 >> max(0, 3 * (depth - 5)))}
    return {"kind": kind, "bits": bits, "depth": rng.randint(4, 5), "chunks": _log_int(rng, 8, 1024)}


# ---- inputs ------------------------------------------------------------------------------------------
def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _noise2(x, z, seed):
    """2D gradient noise (the arithmetic of workloads.perlin2) on the GPU."""
    perm = torch.tensor(W.permutation(int(seed)), dtype=torch.int64, device=x.device)
    grad = torch.tensor([[1, 1], [-1, 1], [1, -1], [-1, -1], [1, 0], [-1, 0], [0, 1], [0, -1]], dtype=torch.float64,
                        device=x.device)
    x0, z0 = torch.floor(x), torch.floor(z)
    xi, zi, xf, zf = x0.long() & 255, z0.long() & 255, x - x0, z - z0
    fade = lambda t: t * t * t * (t * (t * 6.0 - 15.0) + 10.0)  # noqa: E731
    u, v = fade(xf), fade(zf)

    def g(hx, hz, dx, dz):
        k = perm[perm[hx] + hz] & 7
        return grad[k, 0] * dx + grad[k, 1] * dz

    n00, n10 = g(xi, zi, xf, zf), g(xi + 1, zi, xf - 1, zf)
    n01, n11 = g(xi, zi + 1, xf, zf - 1), g(xi + 1, zi + 1, xf - 1, zf - 1)
    a = n00 + u * (n10 - n00)
    return a + v * (n01 + u * (n11 - n01) - a)


def _dtype(bits):
    return torch.uint8 if bits == 8 else torch.int16


def _dunes(chunks, depth, bits, seed, device="cuda"):
    """Dense [chunk][y][z][x] grids of `chunks` dune chunks tiled in XZ (workloads.terrain_params)."""
    side, p = 1 << depth, W.terrain_params(depth)
    nx = max(1, math.isqrt(chunks))
    nz = -(-chunks // nx)
    wx = torch.arange(nx * side, dtype=torch.float64, device=device) / p["scale"]
    wz = torch.arange(nz * side, dtype=torch.float64, device=device) / p["scale"]
    h = p["base"] + torch.floor(p["amp"] * _noise2(wx[None, :].expand(nz * side, -1), wz[:, None].expand(-1, nx * side), seed))
    h = h.to(torch.int16).reshape(nz, side, nx, side).permute(0, 2, 1, 3).reshape(nz * nx, 1, side, side)[:chunks]
    y = torch.arange(side, dtype=torch.int16, device=device)[None, :, None, None]
    out = torch.empty((chunks, side, side, side), dtype=_dtype(bits), device=device)
    step = max(1, (1 << 26) >> (3 * depth))
    for c in range(0, chunks, step):
        d = h[c:c + step] - y
        out[c:c + step] = 3 * (d > 4).to(out.dtype) + 2 * ((d > 1) & (d <= 4)).to(out.dtype) + (d == 1).to(out.dtype)
    return out


def _terrain(case, seed):
    """The world of a case: dune chunks, or one cave tree where a single deep tree is asked for."""
    if case["chunks"] == 1 and case["depth"] >= 7:
        return W.caves_torch(case["depth"], seed=int(seed), device="cuda").to(_dtype(case["bits"]))[None]
    return _dunes(case["chunks"], case["depth"], case["bits"], seed)


def _budget(voxels, floor=64 << 20):
    """Node budget of a program that gives its interner half a byte to a voxel, and never less than 64 MiB."""
    return max(floor, voxels // 2)


def _touch(gen, chunks, depth, density):
    """Per chunk and bottom group (Morton order) the picked voxels as an 8-bit mask [chunks][8^(depth-1)]."""
    groups = 8 ** (depth - 1)
    mask = torch.empty((chunks, groups), dtype=torch.uint8, device="cuda")
    weight = torch.tensor([1 << k for k in range(8)], dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 25) // (8 * groups))
    for c in range(0, chunks, step):
        d = density[c:c + step, None, None]
        pick = torch.rand((d.shape[0], groups, 8), generator=gen, device="cuda") < d
        mask[c:c + step] = (pick.to(torch.uint8) * weight).sum(-1, dtype=torch.uint8)
    return mask


def _records(gen, item0, set_mask, clear_mask, lo, hi):
    """Compacted touched groups of one batch of items (the arrays of vx_apply_groups_async)."""
    at = (set_mask | clear_mask).nonzero()
    s, c = set_mask[at[:, 0], at[:, 1]], clear_mask[at[:, 0], at[:, 1]]
    v = torch.randint(lo, hi + 1, (len(at), 8), generator=gen, device="cuda", dtype=torch.int16)
    bit = (s[:, None] >> torch.arange(8, dtype=torch.uint8, device="cuda")) & 1
    return {"item": (at[:, 0] + item0).to(torch.int32), "group": at[:, 1].to(torch.int32), "set": s, "clear": c,
            "values": v * bit.to(torch.int16)}


def _joined(parts):
    return {k: torch.cat([p[k] for p in parts]).contiguous() for k in parts[0]}


def _split(gen, mask, fraction):
    """Two disjoint masks: each picked voxel goes to the first with probability `fraction`."""
    first = torch.zeros_like(mask)
    for k in range(8):
        first |= (torch.rand(mask.shape, generator=gen, device="cuda") < fraction).to(torch.uint8) << k
    return mask & first, mask & ~first


def _varint_payload(canon, positions, bits):
    """The model payload (leaf table, branch table, chunk records) of a canonical export, in an order that
    depends on the model alone: leaves, then branches from the deepest up."""
    kind = canon["kind"].astype(bool)
    n = len(kind)
    new = np.zeros(n + 1, np.int64)  # new[-1] stays 0: EMPTY
    leaves, branches = np.flatnonzero(kind), np.flatnonzero(~kind)[::-1]
    new[leaves] = 1 + np.arange(len(leaves))
    new[branches] = 1 + len(leaves) + np.arange(len(branches))
    vb = bits // 8

    def stream(columns, varint, keep):
        """Rows of fields to bytes: varint fields in LEB128, the others one byte each."""
        v = columns[keep]
        isv = np.broadcast_to(varint, columns.shape)[keep]
        length = np.ones(len(v), np.int64)
        for k in range(1, 5):
            length += isv & (v >> (7 * k) > 0)
        start = np.cumsum(length) - length
        out = np.zeros(int(length.sum()), np.uint8)
        for k in range(5):
            sel = length > k
            part = np.where(isv[sel], (v[sel] >> (7 * k)) & 0x7F, v[sel] & 0xFF)
            out[start[sel] + k] = part | np.where(isv[sel] & (length[sel] > k + 1), 0x80, 0)
        return out.tobytes()

    value = canon["value"].astype(np.int64)
    be = lambda a: np.stack([(a >> (8 * (vb - 1 - k))) & 0xFF for k in range(vb)], 1)  # noqa: E731
    leaf = np.concatenate([new[leaves][:, None], be(value[leaves])], 1)
    child = new[canon["children"].reshape(n, 8)[branches]]
    branch = np.concatenate([new[branches][:, None], canon["mask"][branches].astype(np.int64)[:, None], child,
                             be(value[branches])], 1)
    keep = np.ones(branch.shape, bool)
    keep[:, 2:10] = child != 0
    u32 = lambda x: int(x).to_bytes(4, "big")  # noqa: E731
    chunks = [u32(len(positions))]
    for (x, y, z), r in zip(positions, canon["roots"]):
        i, b = int(new[r]), b""
        while i >= 0x80:
            b += bytes([i & 0x7F | 0x80])
            i >>= 7
        chunks.append(b"VoxTreeChunk" + b"".join(int(k).to_bytes(4, "big", signed=True) for k in (x, y, z)) + b + bytes([i]))
    return (u32(len(leaves)) + stream(leaf, np.array([True] + [False] * vb), np.ones(leaf.shape, bool)) +
            u32(len(branches)) + stream(branch, np.array([True, False] + [True] * 8 + [False] * vb), keep) + b"".join(chunks))


# ---- a program's handle ---------------------------------------------------------------------------------
def _ptr(t):
    return C.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


class Loaded:
    """An interner on a stream of its own, its trees, and the buffers of one case."""

    def __init__(self, case, budget, patches=0):
        self.case = case
        self.interner = VoxInterner(budget, voxel_bits=case.get("bits", 8), patches=patches)
        self.stream = torch.cuda.Stream()
        self.interner.set_stream(self.stream.cuda_stream)

    def __del__(self):
        if getattr(self, "interner", None) is not None:
            torch.cuda.synchronize()
            self.interner.close()

    def call(self, name, *args):
        self.interner.lib.call(name, self.interner.handle, *args, handle=self.interner.handle)

    def begin(self):
        """The interner's work comes after what the program has queued on its current stream."""
        self.stream.wait_stream(torch.cuda.current_stream())

    def end(self):
        """What the program queues next comes after the interner's work."""
        torch.cuda.current_stream().wait_stream(self.stream)

    def create_trees(self, depths):
        self.depths = np.ascontiguousarray(depths, dtype=np.uint8)
        self.handles = np.zeros(len(depths), np.uint32)
        self.call("trees_create", len(depths), _ptr(self.depths), _ptr(self.handles))
        self.trees = torch.from_numpy(self.handles.view(np.int32)).cuda()

    def build(self, grids, depth, first=0):
        self.begin()
        self.call("build_dense_async", len(grids), C.c_void_p(self.trees.data_ptr() + 4 * first), _ptr(grids), None, depth)
        self.call("interner_sync")

    def read(self, out, depth, first=0):
        self.call("trees_to_dense_async", len(out), C.c_void_p(self.trees.data_ptr() + 4 * first), depth, _ptr(out))

    def apply(self, rec, changed, depth):
        self.call("apply_groups_async", len(self.handles), _ptr(self.trees), _ptr(self.flags), _ptr(self.fill),
                  len(rec["item"]), _ptr(rec["item"]), _ptr(rec["group"]), _ptr(rec["set"]), _ptr(rec["clear"]),
                  _ptr(rec["values"]), _ptr(changed), depth)

    def items(self):
        n = len(self.handles)
        self.flags = torch.full((n,), 2, dtype=torch.uint8, device="cuda")  # patches, no fill
        self.fill = torch.zeros(n, dtype=torch.int32, device="cuda")
        self.changed = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2)]


def _positions(case, seed, count, salt):
    """Random voxel positions of one call (int32 [count][3]), the chunk of each, and the generator."""
    r = np.random.default_rng([int(seed), salt])
    return (r.integers(0, 1 << case["depth"], (count, 3)).astype(np.int32),
            r.integers(0, case["chunks"], count).astype(np.int64), r)


# ---- the kinds of cases -----------------------------------------------------------------------------------
class Points(Loaded):
    """Single-voxel edits: each voxel is placed, then taken away (VoxTree.set / VoxInterner.set_many)."""

    def __init__(self, case, seed):
        n, depth = case["chunks"], case["depth"]
        super().__init__(case, _budget(n << (3 * depth)), EDITING)
        grids = _dunes(n, depth, case["bits"], seed)
        self.objects = [VoxTree(depth) for _ in range(n)]
        host = grids.cpu().numpy()
        self.interner.build_dense(self.objects, host.view(self.interner.dtype))
        self.xyz, chunk, r = _positions(case, seed, case["edits"], 1)
        self.values = r.integers(4, 200, case["edits"]).astype(np.uint32)
        # every voxel is taken away again, and once before the first pass
        self.order = [self.objects[k] for k in chunk] * 2
        self.places = np.concatenate([self.xyz, self.xyz])
        self.writes = np.concatenate([self.values, np.zeros_like(self.values)])
        self.interner.set_many(self.order[:len(chunk)], self.xyz, np.zeros_like(self.values))

    def run(self):
        it = self.interner
        if len(self.values) == 1:
            tree, at, v = self.order[0], tuple(self.xyz[0]), int(self.values[0])
            before = tree.set(it, at, v)
            seen = tree.get(it, at)
            after = tree.set(it, at, 0)
            return {"set": before, "seen": seen or 0, "cleared": after, "then": tree.get(it, at) or 0}
        return {"changed": it.set_many(self.order, self.places, self.writes), "grids": it.to_vec_many(self.objects)}


class Session(Loaded):
    """Whole chunks through the Python classes: clear, dense build, a host Batch, probes, dense read."""

    def __init__(self, case, seed):
        n, depth = case["chunks"], case["depth"]
        super().__init__(case, _budget(n << (3 * depth)), EDITING)
        it = self.interner
        self.grids = _dunes(n, depth, case["bits"], seed).cpu().numpy().view(it.dtype)
        self.objects = [VoxTree(depth) for _ in range(n)]
        self.edits = []
        for k in range(n):
            r = np.random.default_rng([int(seed), 2, k])
            xyz = r.integers(0, 1 << depth, (case["edits"], 3)).astype(np.int32)
            values = r.integers(4, 200, case["edits"]).astype(np.uint32)
            values[r.random(case["edits"]) < 0.15] = 0
            self.edits.append((xyz, values))
        self.batches = [t.create_batch(it) for t in self.objects]

    def run(self):
        it = self.interner
        for t in self.objects:
            t.clear(it)
        built = it.build_dense(self.objects, self.grids)
        for b, (xyz, values) in zip(self.batches, self.edits):
            b.just_clear()
            b.set_many(xyz, values)
        if len(self.objects) == 1:
            applied = self.objects[0].apply_batch(it, self.batches[0])
        else:
            applied = it.apply_batches(self.objects, self.batches)
        probes = self.edits[0][0][:64]
        found, values = it.get_many(np.full(len(probes), self.objects[0].tree, np.uint32), probes)
        return {"built": built, "applied": applied, "found": found, "values": values, "grids": it.to_vec_many(self.objects)}


class Gets(Loaded):
    """Random reads with every argument on the device (vx_get_many_async)."""

    def __init__(self, case, seed):
        n, depth, q = case["chunks"], case["depth"], case["queries"]
        grids = _terrain(case, seed)
        super().__init__(case, _budget(grids.numel()), VX_PATCH_P2)
        self.create_trees([depth] * n)
        self.build(grids, depth)
        self.chunk, self.xyz = _queries(case, seed)
        self.tree = self.trees[self.chunk.long()].contiguous()
        self.found = torch.zeros(q, dtype=torch.uint8, device="cuda")
        self.values = torch.zeros(q, dtype=_dtype(case["bits"]), device="cuda")

    def run(self):
        self.begin()
        self.call("get_many_async", C.c_uint64(len(self.found)), _ptr(self.tree), _ptr(self.xyz), _ptr(self.found),
                  _ptr(self.values))
        self.end()
        return {"found": self.found, "values": self.values}


def _queries(case, seed):
    g = _generator(seed, 3)
    q = case["queries"]
    return (torch.randint(0, case["chunks"], (q,), generator=g, device="cuda", dtype=torch.int32),
            torch.randint(0, 1 << case["depth"], (q, 3), generator=g, device="cuda", dtype=torch.int32))


class Build(Loaded):
    """Every chunk built from its dense grid into an empty interner, and read back dense."""

    def __init__(self, case, seed):
        n, depth = case["chunks"], case["depth"]
        grids = _terrain(case, seed)
        super().__init__(case, _budget(grids.numel()), VX_PATCH_P2)
        self.out = torch.zeros_like(grids)
        if case["host"]:
            self.objects = [VoxTree(depth) for _ in range(n)]
            self.grids = grids.cpu().pin_memory().numpy().view(self.interner.dtype)
        else:
            self.create_trees([depth] * n)
            self.grids = grids
            self.changed = torch.zeros(n, dtype=torch.uint8, device="cuda")

    def run(self):
        depth = self.case["depth"]
        self.begin()
        self.call("interner_reset")
        if self.case["host"]:
            changed = self.interner.build_dense(self.objects, self.grids, mem=VX_MEM_HOST)
            handles = np.array([t.tree for t in self.objects], np.uint32)
            self.call("trees_to_dense", len(handles), _ptr(handles), _ptr(self.out), VX_MEM_DEVICE)
            return {"changed": changed, "grids": self.out}
        self.call("build_dense_async", len(self.changed), _ptr(self.trees), _ptr(self.grids), _ptr(self.changed), depth)
        self.read(self.out, depth)
        self.call("interner_sync")
        self.end()
        return {"changed": self.changed, "grids": self.out}


class Uneven(Loaded):
    """One batched apply of device records over chunks of depths d, d-1 and d-2 (each chunk's density one
    of 1, 1/10, 1/100 of the largest), then one that gives the same voxels other values."""

    def __init__(self, case, seed):
        n, top, bits = case["chunks"], case["depth"], case["bits"]
        self.levels = [top, top - 1, top - 2]
        # both batches' nodes are alive at once while the second one runs
        super().__init__(case, max(64 << 20, 4 * n << (3 * top)), VX_PATCH_P1 | VX_PATCH_P2)
        self.create_trees(np.repeat(self.levels, n))
        gen = _generator(seed, 4)
        density = case["density"] * torch.tensor([0.01, 0.1, 1.0], device="cuda").repeat(n)[:n]
        first, second, self.out = [], [], []
        lo, mid, hi = (4, 100, 255) if bits == 8 else (4, 2000, 4095)
        for k, d in enumerate(self.levels):
            grids = _dunes(n, d, bits, int(seed) + d)
            self.build(grids, d, first=k * n)
            self.out.append(torch.zeros_like(grids))
            picked, cleared = _split(gen, _touch(gen, n, d, density), 0.85)
            first.append(_records(gen, k * n, picked, cleared, lo, mid))
            second.append(_records(gen, k * n, picked, cleared, mid + 1, hi))
        self.records = [_joined(first), _joined(second)]
        self.items()

    def run(self):
        self.begin()
        n, top = self.case["chunks"], self.case["depth"]
        for rec, changed in zip(self.records, self.changed):
            self.apply(rec, changed, top)
        for k, out in enumerate(self.out):
            self.read(out, self.levels[k], first=k * n)
        self.call("interner_maintain")
        self.end()
        return {"changed": self.changed, "grids": self.out}


class Deep(Loaded):
    """Random sets (4 in 5) and clears over one deep cave tree in one apply, then the converse."""

    def __init__(self, case, seed):
        depth, bits = case["depth"], case["bits"]
        grid = _terrain(dict(case, chunks=1), seed)
        super().__init__(case, max(64 << 20, 2 * grid.numel()), VX_PATCH_P1 | VX_PATCH_P2 | VX_PATCH_P3 | VX_PATCH_P4)
        self.create_trees([depth])
        self.build(grid, depth)
        self.out = torch.zeros_like(grid)
        gen = _generator(seed, 5)
        density = torch.full((1,), case["edits"] / float(8 ** depth), device="cuda")
        a, b = _split(gen, _touch(gen, 1, depth, density), 0.8)
        self.records = [_records(gen, 0, a, b, 5, 8), _records(gen, 0, b, a, 5, 8)]
        self.items()

    def run(self):
        self.begin()
        depth = self.case["depth"]
        for rec, changed in zip(self.records, self.changed):
            self.apply(rec, changed, depth)
        self.read(self.out, depth)
        self.call("interner_maintain")
        self.end()
        return {"changed": self.changed, "grid": self.out}


class Serve:
    """A backlog of requests served by voxelis_gb300.serve: sphere fills and reads, then the carves of the
    same spheres and more reads. Spheres sit on a jittered lattice, several to a chunk."""

    def __init__(self, case, seed):
        r = np.random.default_rng([int(seed), 6])
        self.world = World(case["nx"], case["ny"], case["nz"], case["depth"], budget=1 << 30)
        w, side = self.world, self.world.side
        ground = _dunes(case["nx"] * case["nz"], case["depth"], 8, seed)
        trees = w.trees_d[:case["nx"] * case["nz"]].contiguous()
        w.stream.wait_stream(torch.cuda.current_stream())
        w.call("build_dense_async", len(trees), _ptr(trees), _ptr(ground), None, w.depth)
        w.call("interner_sync")
        cells = (case["nx"] * side // 32, case["ny"] * side // 32, case["nz"] * side // 32)
        half = case["edits"] // 2
        at = r.choice(cells[0] * cells[1] * cells[2], half, replace=False)
        fills = []
        for c in at:
            cell = (c % cells[0], c // cells[0] % cells[1], c // (cells[0] * cells[1]))
            center = tuple(int(32 * k + 16 + r.integers(-4, 5)) for k in cell)
            fills.append((center, int(r.integers(2, 12)), int(r.integers(4, 9))))
        spheres = lambda value: [{"kind": EDIT, "t": 0.0, "center": c, "radius": q, "value": v if value else 0,  # noqa: E731
                                  "chunks": sphere_chunks(w, c, q)} for c, q, v in fills]
        size = np.array([case["nx"], case["ny"], case["nz"]]) * side
        pool = [r.integers(0, size, (POINTS_PER_GET, 3)).astype(np.int32) for _ in range(min(8, case["gets"]))]
        reads = [{"kind": GET, "t": 0.0, "pool": k % len(pool)} for k in range(case["gets"])]
        mix = lambda e, g: [x[1] for x in sorted([((i + 0.5) / len(e), x) for i, x in enumerate(e)] +  # noqa: E731
                                                 [((i + 0.25) / max(1, len(g)), x) for i, x in enumerate(g)],
                                                 key=lambda y: y[0])]
        self.requests = mix(spheres(True), reads[::2]) + mix(spheres(False), reads[1::2])
        self.server = Server(w, pool)
        self.server.run(spheres(False), realtime=False)  # the world as every pass finds it

    def __del__(self):
        if getattr(self, "world", None) is not None:
            torch.cuda.synchronize()
            self.world.close()

    def run(self):
        _, results = self.server.run(self.requests, realtime=False, keep_results=True)
        return {"found": np.stack([results[k][0] for k in sorted(results)]),
                "values": np.stack([results[k][1] for k in sorted(results)])}


class Masks(Loaded):
    """Occupancy masks of a world's chunks packed into 64^3 builders (vx_occupancy_masks_async)."""

    def __init__(self, case, seed):
        n, depth = case["chunks"], case["depth"]
        grids = _dunes(n, depth, 8, seed)
        super().__init__(case, _budget(grids.numel()))
        self.create_trees([depth] * n)
        self.build(grids, depth)
        per = 64 >> depth  # chunks a builder takes in x and in z
        self.builders = -(-n // (per * per))
        k = np.arange(n)
        side = 1 << depth
        offsets = np.stack([k % per * side, 0 * k, k // per % per * side], 1).astype(np.int32)
        self.builder_of = torch.from_numpy((k // (per * per)).astype(np.int32)).cuda()
        self.offsets = torch.from_numpy(offsets).cuda()
        b = self.builders
        z = lambda *shape, dtype=torch.int64: torch.zeros(shape, dtype=dtype, device="cuda")  # noqa: E731
        self.out = {"global": z(b, PLANES), "active": z(b, 6), "n": z(b, dtype=torch.int32),
                    "ids": z(b, MAX_MATERIALS, dtype=torch.int32), "counts": z(b, MAX_MATERIALS),
                    "masks": z(b, MAX_MATERIALS, PLANES)}

    def run(self):
        o = self.out
        self.begin()
        self.call("occupancy_masks_async", self.builders, len(self.handles), _ptr(self.trees), _ptr(self.builder_of),
                  _ptr(self.offsets), self.case["depth"], MAX_MATERIALS, _ptr(o["global"]), _ptr(o["active"]), _ptr(o["n"]),
                  _ptr(o["ids"]), _ptr(o["counts"]), _ptr(o["masks"]))
        self.end()
        return o


class Model(Loaded):
    """A model payload loaded into an empty interner (deserialize_model) and written again."""

    def __init__(self, case, seed):
        n, depth = case["chunks"], case["depth"]
        grids = _dunes(n, depth, case["bits"], seed)
        super().__init__(case, _budget(grids.numel(), 256 << 20))
        self.create_trees([depth] * n)
        self.build(grids, depth)
        nx = max(1, math.isqrt(n))
        self.positions = np.array([(k % nx, 0, k // nx) for k in range(n)], np.int32)
        objects = []
        for h in self.handles:
            t = VoxTree(depth)
            t.interner, t.tree = self.interner, int(h)
            objects.append(t)
        self.payload = _varint_payload(self.interner.export_canonical(objects), self.positions, case["bits"])
        self.file = np.zeros(FILE_PER_CHUNK * n + (1 << 16), np.uint8)  # the buffer the model is written to

    def run(self):
        it = self.interner
        self.call("interner_reset")
        trees, positions = it.deserialize_model(self.payload, self.case["depth"])
        blob = it.serialize_model(trees, positions)
        self.file[:len(blob)] = np.frombuffer(blob, np.uint8)
        return {"positions": positions, "size": len(blob), "payload": self.file}


KINDS = {"points": Points, "session": Session, "gets": Gets, "build": Build, "uneven": Uneven, "serve": Serve, "deep": Deep,
         "masks": Masks, "model": Model}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case):
    kind, vb, depth = case["kind"], case.get("bits", 8) // 8, case["depth"]
    grid = vb << (3 * depth)  # bytes of one dense chunk
    n = case.get("chunks", 1)
    if kind == "points":  # position and value in, one flag out, twice
        return {"bytes": 2 * case["edits"] * (12 + vb + 1) + (n * grid if case["edits"] > 1 else 0)}
    if kind == "session":  # grids in and out, the batches' voxels in
        return {"bytes": n * (2 * grid + case["edits"] * (12 + vb))}
    if kind == "gets":  # tree handle and position in, found and value out
        return {"bytes": case["queries"] * (4 + 12 + 1 + vb)}
    if kind == "build":  # grids in, flags out, grids out
        return {"bytes": n * (2 * grid + 1)}
    if kind == "uneven":  # two batches of records in, the grids out
        voxels = sum(n << (3 * (depth - k)) for k in range(3))
        picked = voxels * case["density"] * 1.11 / 3
        groups = min(picked, voxels / 8.0)
        return {"bytes": 2 * groups * (8 + 2 + 8 * vb) + voxels * vb}
    if kind == "deep":
        return {"bytes": 2 * case["edits"] * (8 + 2 + 8 * vb) + grid}
    if kind == "serve":  # points in, found and value out; the spheres' voxels (radius 7 on average), twice
        return {"bytes": case["gets"] * POINTS_PER_GET * 14 + case["edits"] * 1800 * 2}
    if kind == "masks":  # builders out: the three planes and a mask for each material; the chunks come from the tree
        builders = -(-n // ((64 >> depth) ** 2))
        return {"bytes": builders * (PLANES * 8 * (1 + MAX_MATERIALS) + 48 + MAX_MATERIALS * 12)}
    return {"bytes": n * 2 * 300}  # the payload in and out: about 300 bytes for each chunk


def exact(case, seed):
    """The voxels themselves, where a pass returns voxels."""
    if case["kind"] == "gets":
        grids = _terrain(case, seed)
        chunk, xyz = _queries(case, seed)
        v = grids[chunk.long(), xyz[:, 1].long(), xyz[:, 2].long(), xyz[:, 0].long()]
        return {"found": (v != 0).to(torch.uint8), "values": v}
    if case["kind"] == "build":
        grids = _terrain(case, seed)
        changed = (grids.flatten(1) != 0).any(1).to(torch.uint8)
        return {"changed": changed.cpu().numpy() if case["host"] else changed, "grids": grids}
    return None
