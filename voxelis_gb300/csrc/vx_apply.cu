// Batched VoxTree::apply_batch over many trees sharing one interner, level-synchronous on the GPU.
//
// Restates set_batch_at_depth_iterative (spatial/voxtree.rs:724-1118) for n trees at once:
//   plan     the levels' structure from the sorted records alone. A record heads a sibling run at step s
//            (the parents s levels above the bottom groups) when its group differs from the one before it
//            above the 3 s low bits, or it starts an item; counting the records that head each step
//            gives every parent of every level its number, its first child and its first record at once.
//   prep     Phase 0 fill (voxtree.rs:742-758): the fill leaf replaces the old root as the
//            starting node; without patches it is the new root.
//   bottom   Phase 1 (voxtree.rs:770-897), one thread per touched bottom group: descend the old
//            tree to depth d-1, collapse a full uniform group to a leaf, otherwise merge the set
//            voxels into the existing children (or into 8 copies of an ancestor leaf) and
//            hash-cons the branch. The record that heads a parent passes the old node at the parent's
//            place on its descent and leaves it there for the level passes. Groups that change nothing
//            are marked, as the reference drops them.
//   levels   Phase 2 (voxtree.rs:905-1106), one step per level for all trees together: each parent
//            gathers its run's changed children, clones the untouched children of the old parent or
//            replicates an ancestor leaf, collapses 8 equal leaves, and hash-conses the result; a parent
//            none of whose children changed is marked unchanged.
//   finish   apply_batch (voxtree.rs:303-328), by the thread that makes an item's root: commit it,
//            queue the old root for release, report assert_ne!(new_root, old_root) as a reference panic.
// Clear pass (P4). The reference ignores Batch clear bits (voxtree.rs:779). With P4 they are
// honoured as VoxTree::set(pos, 0) for every cleared voxel after the set phase (remove_at_depth,
// voxtree.rs:542-706). Those removals commute, so the same level-synchronous machinery applies them
// in one pass (mode 1): a touched group drops its cleared children (or splits an ancestor leaf into
// 8 copies minus the cleared ones), a parent takes the new children over the old node's children
// (or over 8 copies of an ancestor leaf), clears their types bits, drops children that became
// EMPTY from its mask, and becomes EMPTY itself when its mask empties. Nothing collapses. The
// removal path is refcount-exact, so no correction applies.
// Trees are processed deepest first, so the trees whose root is produced at a step are the tail
// of that step's list, and a parent's number at a step is its number among the records that head it.
//
// Refcounts. After the build every count is the in-degree from newly created nodes plus tree roots,
// plus the corrections below. The lane that creates a branch adds its children's references right
// away, from the key it still holds in registers (no re-read of the node): branch children by a
// global reduction, leaf children into a per-CTA table indexed by leaf value that the CTA flushes
// once (leaves are the hot spots: a few values are named by most bottom groups). The allocation epoch is
// closed once the last level is done. The corrections reproduce where the
// reference's increments differ from the references its nodes hold:
//   Q5 (voxtree.rs:835-839, 846-868): an ancestor leaf is charged 8 - |set| references, but only
//      8 - |modified| slots keep it: + (|modified| - |set|), or + (8 - |set|) when nothing changed.
//   Q6 (voxtree.rs:1062-1072): a collapse with c cloned children gives back min(c, 7) instead of
//      7 - c references: + (7 - 2c).
//   Q7 (voxtree.rs:742-758): the fill leaf's Phase-0 reference is never released when the batch
//      also has patches: + 1.
#include <algorithm>

#include "vx_launch.h"

namespace vxg {
namespace {

constexpr int kThreads = 256;
// minimum resident CTAs of 512 threads the branch-creating kernels are compiled for (2: at most 64
// registers a thread)
#ifndef VX_APPLY_MIN_BLOCKS
#define VX_APPLY_MIN_BLOCKS 2
#endif
__device__ __forceinline__ void add_ref_delta(const DevInterner &I, uint64_t id, int delta) {
    if (delta != 0 && id != EMPTY_ID) atomicAdd(I.refcount + id_index(id), (unsigned)delta);
}

// Per-CTA counts of leaf-child references (dynamic shared memory, leaf_refs_smem bytes). 8-bit
// voxels: one counter per value. 16-bit voxels: kLeafSlots counters direct-mapped by value with the
// owning value as a tag; a value whose slot another value owns goes straight to a global reduction.
constexpr uint32_t kLeafSlots = 4096;
struct LeafRefs {
    uint32_t *cnt;
    uint32_t *tag;  // value + 1 owning the slot, 0 = free (16-bit voxels only)
    uint32_t slots;
    bool direct;
};

__device__ __forceinline__ LeafRefs leaf_refs_init(const DevInterner &I) {
    extern __shared__ uint32_t leaf_smem[];
    LeafRefs L;
    L.direct = I.vbits == 8;
    L.slots = L.direct ? 256u : kLeafSlots;
    L.cnt = leaf_smem;
    L.tag = leaf_smem + L.slots;
    for (uint32_t k = threadIdx.x; k < (L.direct ? L.slots : 2 * L.slots); k += blockDim.x) leaf_smem[k] = 0;
    __syncthreads();
    return L;
}

__device__ __forceinline__ void leaf_ref_add(const DevInterner &I, const LeafRefs &L, uint64_t leaf, uint32_t value,
                                             uint32_t n) {
    if (L.direct) {
        atomicAdd(L.cnt + value, n);
        return;
    }
    const uint32_t s = value & (kLeafSlots - 1u), key = value + 1u;
    uint32_t t = L.tag[s];
    if (t == 0) {
        t = atomicCAS(L.tag + s, 0u, key);
        if (t == 0) t = key;
    }
    if (t == key)
        atomicAdd(L.cnt + s, n);
    else
        atomicAdd(I.refcount + id_index(leaf), n);
}

// One reference per child slot of a node this lane just created (equal children summed first).
__device__ __forceinline__ void add_child_refs(const DevInterner &I, const LeafRefs &L, const uint64_t c[8],
                                               const uint32_t cv[8]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (c[k] == EMPTY_ID) continue;
        bool seen = false;
        uint32_t n = 1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j < k && c[j] == c[k]) seen = true;
            if (j > k && c[j] == c[k]) ++n;
        }
        if (seen) continue;
        if (id_is_leaf(c[k]))
            leaf_ref_add(I, L, c[k], cv[k], n);
        else
            atomicAdd(I.refcount + id_index(c[k]), n);
    }
}

// Adds the CTA's leaf counts to the leaves' global counts (every thread of the CTA calls it).
__device__ __forceinline__ void leaf_refs_flush(const DevInterner &I, const LeafRefs &L) {
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < L.slots; s += blockDim.x) {
        const uint32_t n = L.cnt[s];
        if (n == 0) continue;
        const uint32_t v = L.direct ? s : L.tag[s] - 1u;
        const uint64_t lid = I.leaf_table[v];
        if (lid > LEAF_BUSY)
            atomicAdd(I.refcount + id_index(lid), n);
        else
            set_error(I, ERR_INTERNAL, 47);
    }
}

// ---- items ---------------------------------------------------------------------------------------
// Depth of item i: given by the host, or (check_depths) read from the tree table with the checks of a
// device-resident call. An item that fails them counts as a tree of depth 1, of which no record heads a parent:
// nothing of it is applied.
__device__ __forceinline__ int item_depth_of(const DevInterner &I, const ApplyArgs &a, uint32_t i, bool check_depths,
                                             bool *bad = nullptr) {
    if (!check_depths) return a.it_depth[i];
    const uint32_t t = a.it_tree[i];
    const int d = t < I.tree_cap ? I.depths[t] : TREE_UNUSED;
    int prev = 0xFF;
    if (i > 0) {
        const uint32_t tp = a.it_tree[i - 1];
        prev = tp < I.tree_cap ? I.depths[tp] : TREE_UNUSED;
    }
    if (d == TREE_UNUSED || d > a.max_depth || d < 2 || (i > 0 && d > prev)) {
        if (bad) *bad = true;
        return 1;
    }
    return d;
}

__device__ __forceinline__ uint64_t item_root(const DevInterner &I, const ApplyArgs &a, uint32_t i) {
    const uint32_t t = a.it_tree[i];
    return t < I.tree_cap ? I.roots[t] : EMPTY_ID;
}

// Phase 0 of item i (set phase); refused: it failed the checks of its depth.
__device__ __forceinline__ void prep_item(const DevInterner &I, const ApplyArgs &a, uint32_t i, bool refused) {
    const uint64_t old = item_root(I, a, i);
    const uint8_t f = a.it_flags[i];
    uint64_t init = old;
    a.it_old[i] = old;
    a.it_panic[i] = refused;
    a.it_changed[i] = 0;
    if ((f & 1) && !refused) {
        bool created;
        const uint64_t fill = intern_leaf(I, a.it_fill[i], &created);
        init = fill;
        if (f & 2) add_ref_delta(I, fill, 1);  // Q7
    }
    a.it_init[i] = init;
}

// Whether item i has records: by the host's counts, or by a search in the sorted records of a device-resident call.
__device__ __forceinline__ bool item_has_records(const ApplyArgs &a, uint32_t i) {
    if (a.it_first) return a.it_first[i] < a.it_first[i + 1];
    uint32_t lo = 0, hi = a.n_records;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (a.rec_item[mid] < i)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo < a.n_records && a.rec_item[lo] == i;
}

// The root of item i is nw (mode 0: the set phase, voxtree.rs:303-328; mode 1: the clear pass). Once an item and
// mode, whatever the records are (release_list has a place for each, and a root is released once): the first to
// come takes the item's word, it_old of the set phase and it_init of the clear pass. Records in order name an item's
// root once; others are an error.
__device__ __forceinline__ void finish_item(const DevInterner &I, const ApplyArgs &a, int mode, uint32_t i, uint64_t nw) {
    const uint32_t t = a.it_tree[i];
    if (t >= I.tree_cap || (mode == 0 && a.it_panic[i])) return;
    uint64_t old = atomicExch((unsigned long long *)(mode ? a.it_init : a.it_old) + i, INVALID_ID);
    if (old == INVALID_ID) {
        set_error(I, ERR_INVALID, 48);
        return;
    }
    if (mode == 1) {
        old = I.roots[t];
        if (nw != EMPTY_ID) atomicAdd(I.refcount + id_index(nw), 1u);
    } else {
        if ((a.it_flags[i] & 3) && nw != EMPTY_ID) atomicAdd(I.refcount + id_index(nw), 1u);  // the tree's root reference
        if (old != EMPTY_ID && nw == old && !(I.flags & (1u << 4))) {  // assert_ne!(new_root_id, self.root_id) (voxtree.rs:311)
            set_error(I, ERR_REF_PANIC, 41);
            return;
        }
    }
    if (old != EMPTY_ID) {
        const unsigned long long e = atomicAdd(&I.ctr->scratch[SC_RELEASE], 1ull);
        a.release_list[e] = old;
    }
    I.roots[t] = nw;
    a.it_changed[i] = 1;
}

// ---- the plan of the levels ------------------------------------------------------------------------
// Records are taken in tiles of 32 (one warp). The CTAs of the grid own contiguous ranges of tiles, their
// warps contiguous parts of a range. Word 0 of a count is the records with clear bits, word s the records
// that head step s, word kRootWord + s the items whose root is made at step s; lane s of a warp keeps word s.
struct Tiles {
    uint32_t total, per_cta, per_warp;
    __device__ explicit Tiles(const ApplyArgs &a) {
        const uint32_t nw = blockDim.x >> 5;
        total = (uint32_t)(((uint64_t)a.n_records + 31) / 32);
        per_cta = (total + gridDim.x - 1) / gridDim.x;
        per_warp = (per_cta + nw - 1) / nw;
    }
    // This warp's tiles [lo, hi).
    __device__ void own(uint32_t *lo, uint32_t *hi) const {
        const uint32_t warp = threadIdx.x >> 5;
        const uint64_t c0 = (uint64_t)blockIdx.x * per_cta, c1 = c0 + per_cta < total ? c0 + per_cta : total;
        const uint64_t w0 = c0 + (uint64_t)warp * per_warp, w1 = w0 + per_warp < c1 ? w0 + per_warp : c1;
        *lo = (uint32_t)(w0 < w1 ? w0 : 0);
        *hi = (uint32_t)(w0 < w1 ? w1 : 0);
    }
    // Place in ApplyArgs::warp_off of the warp that counted the tile.
    __device__ uint32_t off(uint32_t tile) const {
        const uint32_t c = tile / per_cta;
        return (c * (blockDim.x >> 5) + (tile - c * per_cta) / per_warp) * kPlanWords;
    }
};

// Whether a tree of depth d has bottom group g.
__device__ __forceinline__ bool group_in_tree(uint32_t g, int d) { return g >> (3 * (d - 1)) == 0; }

// Steps that record r (of item i and group g, depth d) heads: 1 .. the result, none for a group outside the tree.
// The one of an item that heads all d - 1 is its first. Whole warp, lanes in order.
__device__ __forceinline__ uint32_t head_steps(const ApplyArgs &a, uint64_t r, bool in, uint32_t i, uint32_t g, int d) {
    uint32_t ip = __shfl_up_sync(0xFFFFFFFFu, i, 1), gp = __shfl_up_sync(0xFFFFFFFFu, g, 1);
    if (!in || !group_in_tree(g, d)) return 0;
    const uint32_t top = (uint32_t)d - 1u;
    if ((threadIdx.x & 31u) == 0 && r > 0) {
        ip = a.rec_item[r - 1];
        gp = a.rec_group[r - 1];
    }
    if (r == 0 || ip != i) return top;
    const uint32_t x = g ^ gp, s = x ? (31u - __clz(x)) / 3u : 0u;
    return s < top ? s : top;
}

// Counts of this CTA's range (all threads of the CTA call it; cnt_s: kPartWords words a warp).
__device__ __forceinline__ void plan_count(const DevInterner &I, const ApplyArgs &a, bool check_depths,
                                           uint32_t (*cnt_s)[kPartWords]) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t lo, hi;
    Tiles(a).own(&lo, &hi);
    uint32_t acc = 0;  // word `lane`, over this warp's tiles so far
    for (uint32_t tile = lo; tile < hi; ++tile) {
        const uint64_t r = 32ull * tile + lane;
        const bool in = r < a.n_records;
        const uint32_t i = in ? a.rec_item[r] : 0u, g = in ? a.rec_group[r] : 0u;
        const int d = in ? item_depth_of(I, a, i, check_depths) : 2;
        const uint32_t hs = head_steps(a, r, in, i, g, d);
        if (lane < kPlanWords) a.tile_base[(uint64_t)tile * kPlanWords + lane] = acc;
        // the first record of an item heads every step up to its root's
        for (unsigned h = __ballot_sync(0xFFFFFFFFu, hs && hs == (uint32_t)d - 1u); h; h &= h - 1) {
            const uint32_t root_step = __shfl_sync(0xFFFFFFFFu, hs, __ffs(h) - 1);
            if (lane == kRootWord + root_step) ++acc;
        }
        const unsigned cl = __ballot_sync(0xFFFFFFFFu, in && a.rec_clear[r] != 0);
        if (lane == 0) acc += __popc(cl);
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, hs);
        for (uint32_t s = 1; s <= top; ++s) {
            const unsigned b = __ballot_sync(0xFFFFFFFFu, hs >= s);
            if (lane == s) acc += __popc(b);
        }
    }
    if (lane < kPartWords) cnt_s[warp][lane] = acc;
    __syncthreads();
    if (threadIdx.x < kPartWords) {  // the warps' places in the range, and its sums
        uint32_t run = 0;
        for (uint32_t w = 0; w < nw; ++w) {
            if (threadIdx.x < kPlanWords) a.warp_off[(blockIdx.x * nw + w) * kPlanWords + threadIdx.x] = run;
            run += cnt_s[w][threadIdx.x];
        }
        a.part[threadIdx.x * gridDim.x + blockIdx.x] = run;
    }
    __syncthreads();
}

struct Plan {
    uint32_t base[kPlanWords];   // counts of the ranges before this CTA's
    uint32_t total[kPartWords];  // counts of all ranges, no more than a step's room
};
// From this many tiles a warp on, the bottom groups are shared out in turn (bottom_records): a range of
// neighbouring records is as dense or as new as its part of the world, and the CTAs with the heaviest ranges
// were awaited for a fifth of the bottom's time. In turn against in ranges, an apply of trees of depth 7: 2456
// against 2710 us for 6.3 M records, 707 against 719 for 1.16 M; from a tile a warp on, 393 against 384 for
// 0.29 M: the barrier behind the places.
constexpr uint32_t kTurnTiles = 4;
__device__ __forceinline__ bool tiles_in_turn(const ApplyArgs &a) {
    return a.n_records >= (uint64_t)kTurnTiles * gridDim.x * blockDim.x;
}

// Entries of step s - 1 (records for s = 1) that have a parent at step s: all but the roots, which are the
// tail of the list.
__device__ __forceinline__ uint32_t plan_children(const ApplyArgs &a, const uint32_t *total, uint32_t s) {
    if (s == 1) return a.n_records;
    const uint32_t n = total[s - 1], roots = total[kRootWord + s - 1];
    return n > roots ? n - roots : 0;
}

// After every CTA's plan_count: the totals, and (places, once) this CTA's warps' places among all records. All
// threads of the CTA call it.
__device__ __forceinline__ void plan_totals(const ApplyArgs &a, Plan &P, bool places = true) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t s = warp; s < kPartWords; s += nw) {
        uint32_t before = 0, all = 0;
        for (uint32_t c = lane; c < gridDim.x; c += 32) {
            const uint32_t v = a.part[s * gridDim.x + c];
            all += v;
            if (c < blockIdx.x) before += v;
        }
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        all = __reduce_add_sync(0xFFFFFFFFu, all);
        if (lane == 0) {
            if (s < kPlanWords) P.base[s] = before;
            P.total[s] = s > 0 && s < kPlanWords && all > a.p_cap[s] ? a.p_cap[s] : all;
        }
    }
    __syncthreads();
    if (!places) return;
    for (uint32_t k = threadIdx.x; k < nw * kPlanWords; k += blockDim.x)
        a.warp_off[blockIdx.x * nw * kPlanWords + k] += P.base[k % kPlanWords];
    __syncthreads();
}

// ---- Phase 1 -----------------------------------------------------------------------------------------
// An entry's value word: LOD value, the slot among its siblings, and whether it changed.
constexpr uint32_t kChanged = 1u << 31;
__device__ __forceinline__ uint32_t entry_word(uint32_t value, uint32_t path, bool changed) {
    return value | ((path & 7u) << 16) | (changed ? kChanged : 0u);
}

// The records of this warp's tiles: those it counted, or (in_turn, once every CTA has been through plan_totals)
// every so many tiles of the whole. In the set phase it also writes the parents' first children and records; in
// both the old node at each parent's place.
__device__ __forceinline__ void bottom_records(const DevInterner &I, const ApplyArgs &a, int mode, const LeafRefs &L,
                                               bool in_turn) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt = (1u << lane) - 1u;
    const Tiles tiles(a);
    uint32_t lo, hi, step = 1;
    tiles.own(&lo, &hi);
    if (in_turn) {
        lo = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        hi = tiles.total;
        step = gridDim.x * blockDim.x >> 5;
    }
    for (uint32_t tile = lo; tile < hi; tile += step) {
        const uint64_t r = 32ull * tile + lane;
        const bool in = r < a.n_records;
        const uint32_t i = in ? a.rec_item[r] : 0u, g = in ? a.rec_group[r] : 0u;
        const int d = in ? a.it_depth[i] : 2;
        const uint32_t hs = head_steps(a, r, in, i, g, d);
        const uint32_t at = lane < kPlanWords ? a.warp_off[tiles.off(tile) + lane] + a.tile_base[(uint64_t)tile * kPlanWords + lane] : 0u;
        bool active = in;
        uint32_t set = 0, changed = 0;
        uint64_t cur = EMPTY_ID, anc = EMPTY_ID, out = EMPTY_ID;
        uint32_t v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint64_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t cv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t types = 0, mask = 0, lod = 0;
        bool want_branch = false;
        if (in) {
            set = mode ? a.rec_clear[r] : a.rec_set[r];
            if (set == 0 || a.it_panic[i]) active = false;
            if (!group_in_tree(g, d)) {
                set_error(I, ERR_INVALID, 49);
                active = false;
            }
        }
        if (active || hs) cur = mode ? item_root(I, a, i) : a.it_init[i];
        // descend to depth d-1 (voxtree.rs:792-822); at step s the node is the old one of the parent there
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, in ? (uint32_t)d - 1u : 0u);
        uint32_t above = 0;  // this record's number at step s + 1, when it heads it
        for (uint32_t s = top; s >= 1; --s) {
            const unsigned b = __ballot_sync(0xFFFFFFFFu, hs >= s);
            const uint32_t p = __shfl_sync(0xFFFFFFFFu, at, s) + __popc(b & lt);
            if (hs > s && mode == 0 && above < a.p_cap[s + 1]) a.p_start[s + 1][above] = p;
            if (hs >= s) {
                if (p < a.p_cap[s]) {
                    a.p_old[s][p] = anc != EMPTY_ID ? anc : cur;
                    if (mode == 0) a.p_rec[s][p] = (uint32_t)r;
                } else {
                    set_error(I, ERR_INVALID, 47);  // records that are not sorted by (item, group)
                }
                above = p;
            }
            if (s < (uint32_t)d && cur != EMPTY_ID) {
                if (id_is_branch(cur)) {
                    cur = I.children[8ull * id_index(cur) + ((g >> (3 * (s - 1))) & 7u)];
                } else {
                    anc = cur;
                    cur = EMPTY_ID;
                }
            }
        }
        if (hs && mode == 0 && above < a.p_cap[1]) a.p_start[1][above] = (uint32_t)r;
        bool uniform = false;
        if (active) {
            if ((reinterpret_cast<uintptr_t>(a.rec_vals) & 15u) == 0) {
                const uint4 w = reinterpret_cast<const uint4 *>(a.rec_vals)[r];
                const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = (ws[k >> 1] >> (16 * (k & 1))) & 0xFFFFu;
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = a.rec_vals[8 * r + k];
            }
            uniform = set == 0xFF;
#pragma unroll
            for (int k = 1; k < 8; ++k) uniform = uniform && v[k] == v[0];
            if (cur != EMPTY_ID && id_is_leaf(cur)) {
                if ((I.flags & 1u) || mode == 1) {  // P1 (removals always split a leaf)
                    anc = cur;
                    cur = EMPTY_ID;
                } else if (!uniform) {  // the reference panics in BlockId::types()
                    a.it_panic[i] = 1;
                    set_error(I, ERR_REF_PANIC, 40);
                    active = false;
                }
            }
        }
        if (active && mode == 1) {  // remove_at_depth_branch / _leaf at depth d-1
            uint32_t modified = 0;
            if (cur != EMPTY_ID) {
                const uint64_t *src = I.children + 8ull * id_index(cur);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    c[k] = src[k];
                    cv[k] = c[k] ? node_value(I, id_index(c[k])) : 0;
                }
                types = id_types(cur);
                mask = id_mask(cur);
                modified = set & mask;
            } else if (anc != EMPTY_ID) {
                const uint32_t av = node_value(I, id_index(anc));
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    c[k] = anc;
                    cv[k] = av;
                }
                types = mask = 0xFF;
                modified = set;
            }
            if (modified) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if ((modified >> k) & 1) {
                        c[k] = EMPTY_ID;
                        cv[k] = 0;
                    }
                types &= ~modified;
                mask &= ~modified;
                changed = 1;
                if (mask) want_branch = true;
            }
        } else if (active && uniform) {  // voxtree.rs:826, 887-896
            bool created;
            out = intern_leaf(I, v[0], &created);
            lod = v[0];
            changed = 1;
        } else if (active) {  // voxtree.rs:829-883
            if (cur != EMPTY_ID) {
                const uint64_t *src = I.children + 8ull * id_index(cur);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    c[k] = src[k];
                    cv[k] = c[k] ? node_value(I, id_index(c[k])) : 0;
                }
                types = id_types(cur);
                mask = id_mask(cur);
            } else if (anc != EMPTY_ID) {
                const uint32_t av = node_value(I, id_index(anc));
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    c[k] = anc;
                    cv[k] = av;
                }
                types = mask = 0xFF;
            }
            // the set voxels whose value differs from the existing leaf become new leaves: their
            // leaf-table slots are read together (one round trip for all of them); only a leaf not
            // created yet takes the claiming path
            uint32_t modified = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (((set >> k) & 1) && !(c[k] != EMPTY_ID && cv[k] == v[k])) modified |= 1u << k;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if ((modified >> k) & 1) c[k] = ld_cg(I.leaf_table + v[k]);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (!((modified >> k) & 1)) continue;
                if (c[k] <= LEAF_BUSY) {
                    bool created;
                    c[k] = intern_leaf(I, v[k], &created);
                }
                cv[k] = v[k];
            }
            types |= modified;
            mask |= modified;
            if (anc != EMPTY_ID && cur == EMPTY_ID) {  // Q5
                const int ds = __popc(set), dm = __popc(modified);
                add_ref_delta(I, anc, modified ? dm - ds : 8 - ds);
            }
            if (modified) {
                want_branch = true;
                changed = 1;
            }
        }
        bool created;
        const uint64_t id = warp_intern_branch_inl(I, want_branch, c, types, mask, [&] {
            if (want_branch) lod = calc_average8(cv);
            return lod;
        }, &created);
        if (created) add_child_refs(I, L, c, cv);
        if (want_branch) out = id;
        if (in) {
            a.rec_id[r] = out;
            a.rec_val[r] = entry_word(lod, g, changed != 0);
        }
    }
}

// ---- Phase 2 -----------------------------------------------------------------------------------------
// Parents cta_base + threadIdx.x, + stride, ... of step s (n_par of them, their children are the first n_child
// entries of step s - 1). A CTA-uniform loop: whole warps take part in the warp-cooperative interning.
__device__ __forceinline__ void parents_range(const DevInterner &I, const ApplyArgs &a, int mode, const LeafRefs &L,
                                              uint32_t s, uint32_t n_par, uint32_t n_child, uint64_t cta_base, uint64_t stride) {
    const uint64_t *in_id = s == 1 ? a.rec_id : a.e_id[(s - 1) & 1];
    const uint32_t *in_val = s == 1 ? a.rec_val : a.e_val[(s - 1) & 1];
    for (uint64_t base = cta_base; base < n_par; base += stride) {
        const uint64_t p = base + threadIdx.x;
        const bool in = p < n_par;
        uint64_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t cv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        uint32_t types = 0, mask = 0;
        uint32_t i = 0, path = 0, d = 0;
        bool want_branch = false, changed = false;
        uint64_t out = EMPTY_ID;
        uint32_t out_val = 0;
        if (in) {
            const uint32_t r0 = a.p_rec[s][p];
            i = a.rec_item[r0];
            path = a.rec_group[r0] >> (3 * s);
            d = a.it_depth[i];
            const uint32_t b = a.p_start[s][p];
            uint32_t e = p + 1 < n_par ? a.p_start[s][p + 1] : n_child;
            if (e > n_child) e = n_child;
            // gather the run of changed children (voxtree.rs:959-1000), four loads in flight; slots by
            // select, so that the arrays stay in registers
            for (uint32_t j0 = b; j0 < e; j0 += 4) {
                uint32_t ev[4];
                uint64_t id[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    ev[q] = j0 + q < e ? in_val[j0 + q] : 0u;
                    id[q] = j0 + q < e ? in_id[j0 + q] : 0ull;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!(ev[q] & kChanged)) continue;
                    const uint32_t ti = (ev[q] >> 16) & 7u;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if ((uint32_t)k == ti) {
                            c[k] = id[q];
                            cv[k] = ev[q] & 0xFFFFu;
                        }
                    types |= (id_is_leaf(id[q]) ? 1u : 0u) << ti;
                    mask |= 1u << ti;
                }
            }
            changed = mask != 0;
        }
        if (changed) {
            // the old node at the parent's place (voxtree.rs:934-952): a branch, or a leaf at or above it
            uint64_t eq = a.p_old[s][p], leaf = EMPTY_ID;
            if (id_is_leaf(eq)) {
                leaf = eq;
                eq = EMPTY_ID;
            }
            if (mode == 1) {  // remove_at_depth_branch / _leaf one level up (voxtree.rs:559-706)
                const uint32_t ch = mask;
                uint64_t nc[8];
                uint32_t nv[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    nc[k] = c[k];
                    nv[k] = cv[k];
                }
                if (eq != EMPTY_ID) {
                    const uint64_t *src = I.children + 8ull * id_index(eq);
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        c[k] = src[k];
                        cv[k] = c[k] ? node_value(I, id_index(c[k])) : 0;
                    }
                    types = id_types(eq) & ~ch;
                    mask = id_mask(eq);
                } else if (leaf != EMPTY_ID) {
                    const uint32_t lv = node_value(I, id_index(leaf));
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        c[k] = leaf;
                        cv[k] = lv;
                    }
                    types = 0xFFu & ~ch;
                    mask = 0xFF;
                } else {
                    set_error(I, ERR_INTERNAL, 45);
                    types = 0;
                    mask = 0;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if ((ch >> k) & 1) {
                        c[k] = nc[k];
                        cv[k] = nv[k];
                        if (nc[k] == EMPTY_ID)
                            mask &= ~(1u << k);
                        else
                            mask |= 1u << k;
                    }
                if (mask) want_branch = true;
            } else {
                const uint32_t existing_mask = eq != EMPTY_ID ? id_mask(eq) : 0u;
                const uint32_t inv = (~mask) & 0xFFu;
                const uint32_t cloned = existing_mask & inv;
                if (mask != 0xFF) {
                    if (cloned) {  // voxtree.rs:1017-1031
                        const uint64_t *src = I.children + 8ull * id_index(eq);
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            if (!((cloned >> k) & 1)) continue;
                            c[k] = src[k];
                            cv[k] = c[k] ? node_value(I, id_index(c[k])) : 0;
                            types |= (id_is_leaf(c[k]) ? 1u : 0u) << k;
                            mask |= 1u << k;
                        }
                    } else if (leaf != EMPTY_ID) {  // voxtree.rs:1032-1047
                        const uint32_t lv = node_value(I, id_index(leaf));
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if ((inv >> k) & 1) {
                                c[k] = leaf;
                                cv[k] = lv;
                            }
                        types |= inv;
                        mask |= inv;
                    }
                }
                bool same = types == 0xFF;
#pragma unroll
                for (int k = 1; k < 8; ++k) same = same && c[k] == c[0];
                if (same) {  // voxtree.rs:1062-1075
                    out = c[0];
                    out_val = cv[0];
                    if (cloned) add_ref_delta(I, c[0], 7 - 2 * __popc(cloned));  // Q6
                } else {
                    want_branch = true;
                }
            }
        }
        bool created;
        const uint64_t id = warp_intern_branch_inl(I, want_branch, c, types, mask, [&] {
            if (want_branch) out_val = calc_average8(cv);
            return out_val;
        }, &created);
        if (created) add_child_refs(I, L, c, cv);
        if (!in) continue;
        if (want_branch) out = id;
        if (d - 1u == s) {  // (a fill without the patches bit is the root that unchanged records leave)
            if (changed || (mode == 0 && !(a.it_flags[i] & 2))) finish_item(I, a, mode, i, changed ? out : a.it_init[i]);
            a.e_val[s & 1][p] = 0;  // no entry of the next step's (records out of order may leave it within a run)
        } else {
            a.e_id[s & 1][p] = out;
            a.e_val[s & 1][p] = entry_word(out_val, path, changed);
        }
    }
}

// ---- phases of an apply ------------------------------------------------------------------------------
// Set phase: depths, Phase 0 and the counts of the plan. All threads of the grid.
__device__ __forceinline__ void phase_plan(const DevInterner &I, const ApplyArgs &a, bool check_depths,
                                           uint32_t (*cnt_s)[kPartWords]) {
    const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (gt == 0) I.ctr->scratch[SC_RELEASE] = 0;
    for (uint64_t i = gt; i < a.n_items; i += stride) {
        bool bad = false;
        if (check_depths) {
            const_cast<uint8_t *>(a.it_depth)[i] = (uint8_t)item_depth_of(I, a, (uint32_t)i, true, &bad);
            if (bad) set_error(I, ERR_INVALID, 46);
        }
        prep_item(I, a, (uint32_t)i, bad);
    }
    plan_count(I, a, check_depths, cnt_s);
}

// Phase 1, and the roots of the items without patches and records.
__device__ __forceinline__ void phase_bottom(const DevInterner &I, const ApplyArgs &a, int mode, const LeafRefs &L,
                                             bool in_turn) {
    const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (mode == 0)
        for (uint64_t i = gt; i < a.n_items; i += stride)
            if (!(a.it_flags[i] & 2) && !item_has_records(a, (uint32_t)i)) finish_item(I, a, 0, (uint32_t)i, a.it_init[i]);
    bottom_records(I, a, mode, L, in_turn);
}

// Whether the release of the roots that the set phase replaced can wait for the clear pass and go with its own,
// which leaves out half of the release rounds (an apply of a tree of depth 9 541 us against 577 for 261 K records,
// 301 against 363 for 16 K). Counts are sums and no count that the set phase left can fall before, so only the free
// nodes decide: what the clear pass can make at most has to be free without the set phase's dead. One thread, after
// the set phase's epoch is closed.
__device__ bool release_can_wait(const DevInterner &I, const uint32_t *total, int max_depth) {
    if (total[0] == 0) return false;  // no clear pass
    uint64_t most = total[0];
    for (int s = 1; s <= max_depth - 1; ++s) most += total[s];
    return most <= (uint64_t)I.capacity - I.ctr->next_index + I.ctr->free_count;
}

constexpr int kMaxApplyWarps = 16;  // 512 threads

// One launch per phase (tune_set_launch 0).
__global__ void __launch_bounds__(512) apply_plan_kernel(DevInterner I, ApplyArgs a, int check_depths) {
    pdl_wait();
    pdl_release();
    __shared__ uint32_t cnt_s[kMaxApplyWarps][kPartWords];
    phase_plan(I, a, check_depths != 0, cnt_s);
}

__global__ void __launch_bounds__(512, VX_APPLY_MIN_BLOCKS) apply_bottom_kernel(DevInterner I, ApplyArgs a, int mode) {
    pdl_wait();
    pdl_release();
    __shared__ Plan P;
    plan_totals(a, P, mode == 0);
    if (blockIdx.x == 0 && threadIdx.x < kPartWords) a.level_n[threadIdx.x] = P.total[threadIdx.x];
    if (mode == 1 && blockIdx.x == 0 && threadIdx.x == 0 && !I.ctr->scratch[SC_DEFER]) I.ctr->scratch[SC_RELEASE] = 0;
    if (mode == 0 || P.total[0]) {
        const LeafRefs L = leaf_refs_init(I);
        phase_bottom(I, a, mode, L, false);
        leaf_refs_flush(I, L);
    }
    // without records no level pass follows that would close the epoch
    if (a.n_records == 0 && grid_last_cta(&I.ctr->scratch[SC_DONE])) {
        epoch_finalize_body(I);
        I.ctr->scratch[SC_DEFER] = 0;
    }
}

__global__ void __launch_bounds__(512, VX_APPLY_MIN_BLOCKS) apply_parents_kernel(DevInterner I, ApplyArgs a, int mode, int s,
                                                                                 int clear_follows) {
    pdl_wait();
    pdl_release();
    if (mode == 0 || a.level_n[0]) {
        const LeafRefs L = leaf_refs_init(I);
        parents_range(I, a, mode, L, s, a.level_n[s], plan_children(a, a.level_n, s),
                      (uint64_t)blockIdx.x * blockDim.x, (uint64_t)gridDim.x * blockDim.x);
        leaf_refs_flush(I, L);
    }
    if (s == a.max_depth - 1 && grid_last_cta(&I.ctr->scratch[SC_DONE])) {
        epoch_finalize_body(I);
        I.ctr->scratch[SC_DEFER] = clear_follows && release_can_wait(I, a.level_n, a.max_depth);
    }
}

// ---- the whole apply in one launch ---------------------------------------------------------------------
// One cluster: its hardware barrier, in the form that a warp's threads may come to apart (phases end behind
// branches of single threads).
struct ClusterBarrier {
    __device__ explicit ClusterBarrier(const DevInterner &) {}
    __device__ bool usable() { return true; }
    __device__ bool sync() {
        asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
    __device__ void leave() {}
};

// The set phase (mode 0) and, when `clear_pass` and some record has clear bits, the clear pass (mode 1), each
// with its release: the phases of the separate launches with a barrier after each. Barriers: two, one a
// level, one for the roots and one a release round that has nodes.
template <class Barrier>
__device__ __forceinline__ void apply_single(const DevInterner &I, const ApplyArgs &a, int check_depths, int clear_pass,
                                             uint32_t *frontier_a, uint32_t *frontier_b, int rounds) {
    extern __shared__ uint32_t leaf_smem[];
    __shared__ uint32_t cnt_s[kMaxApplyWarps][kPartWords];
    __shared__ Plan P;
    const uint64_t cta_base = (uint64_t)blockIdx.x * blockDim.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const bool t0 = cta_base + threadIdx.x == 0;
    DevCounters *ctr = I.ctr;
    Barrier bar(I);
    if (!bar.usable()) return;
    phase_plan(I, a, check_depths != 0, cnt_s);
    if (!bar.sync()) return;
    plan_totals(a, P);
    const bool in_turn = tiles_in_turn(a);
    if (in_turn && !bar.sync()) return;
    bool deferred = false;  // the same in every thread
    for (int mode = 0; mode <= clear_pass && (mode == 0 || P.total[0]); ++mode) {
        const LeafRefs L = leaf_refs_init(I);
        if (t0) {  // (nothing reads them before the barrier after the last level)
            ctr->rel_count[0] = ctr->rel_count[1] = ctr->rel_count[2] = 0;
            if (mode == 1 && !deferred) ctr->scratch[SC_RELEASE] = 0;
        }
        phase_bottom(I, a, mode, L, in_turn);
        if (!bar.sync()) return;
        for (int s = 1; s <= a.max_depth - 1 && a.n_records; ++s) {
            parents_range(I, a, mode, L, s, P.total[s], plan_children(a, P.total, s), cta_base, stride);
            if (s == a.max_depth - 1) leaf_refs_flush(I, L);
            if (!bar.sync()) return;
        }
        if (mode == 0 && clear_pass && P.total[0]) {
            if (t0) {
                epoch_finalize_body(I);
                ctr->scratch[SC_DEFER] = release_can_wait(I, P.total, a.max_depth);
                ctr->scratch[SC_FREE_BASE] = ctr->free_count;
            }
            if (!bar.sync()) return;
            deferred = *(volatile unsigned long long *)&ctr->scratch[SC_DEFER] != 0;
            if (deferred) continue;
        } else if (t0) {
            epoch_finalize_body(I);
            ctr->scratch[SC_FREE_BASE] = ctr->free_count;
        }
        release_roots_range(I, a.release_list, frontier_a, &ctr->rel_count[0], cta_base, stride);
        const LeafDrops D = leaf_drops_init(I, leaf_smem);  // the leaf counts were flushed before the last barrier
        if (!bar.sync()) return;
        // round r reads set r % 3 and writes set (r + 1) % 3; set (r + 2) % 3 was read by round r - 1
        // and is written by round r + 1, so it is cleared now
        uint32_t *fr[2] = {frontier_a, frontier_b};
        uint64_t free_base = *(volatile unsigned long long *)&ctr->scratch[SC_FREE_BASE];
        for (int r = 0; r < rounds; ++r) {
            const uint64_t n = *(volatile unsigned long long *)&ctr->rel_count[r % 3];
            if (n == 0) break;  // the same answer in every CTA
            if (t0) ctr->rel_count[(r + 2) % 3] = 0;
            release_round_range(I, D, fr[r & 1], fr[(r + 1) & 1], n, free_base, &ctr->rel_count[(r + 1) % 3], cta_base, stride);
            free_base += n;
            if (!bar.sync()) return;
        }
    }
    if (t0) ctr->rel_count[0] = ctr->rel_count[1] = ctr->rel_count[2] = 0;  // as the release launches expect
    bar.leave();
}

// 80 registers, three CTAs of 256 an SM: 34 bytes of spills a thread. With 64 (four CTAs, 180 bytes of spills a thread) 6.3 M bottom
// groups took 2453 us against 2379, 580 K 502 against 472, 32 K of a tree of depth 9 381 against 375; with 96 (two
// CTAs) 2663, 505 and 373.
__global__ void __maxnreg__(80) apply_grid_kernel(const DevInterner I, const ApplyArgs a,
                                                                              int check_depths, int clear_pass,
                                                                              uint32_t *frontier_a, uint32_t *frontier_b,
                                                                              int rounds) {
    apply_single<GridBarrier>(I, a, check_depths, clear_pass, frontier_a, frontier_b, rounds);
}

__global__ void __launch_bounds__(512, 1) apply_cluster_kernel(const DevInterner I, const ApplyArgs a, int check_depths,
                                                               int clear_pass, uint32_t *frontier_a, uint32_t *frontier_b,
                                                               int rounds) {
    apply_single<ClusterBarrier>(I, a, check_depths, clear_pass, frontier_a, frontier_b, rounds);
}

// rec_item[r] = i for every record r of item i (records of item i: [first[i], first[i+1])), one CTA
// per item with coalesced stores.
__global__ void __launch_bounds__(kThreads) expand_items_kernel(const uint32_t *first, uint32_t n,
                                                               uint32_t *rec_item) {
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
        const uint32_t r1 = first[i + 1];
        for (uint32_t r = first[i] + threadIdx.x; r < r1; r += blockDim.x) rec_item[r] = i;
    }
}

}  // namespace

// Dynamic shared memory of the kernels that create branches (their LeafRefs table), and of the single
// launch, whose release rounds use it in turn.
static size_t leaf_refs_smem(const DevInterner &I) { return I.vbits == 8 ? 256 * 4 : 2 * kLeafSlots * 4; }

static int apply_threads_of(const ApplyArgs &a) { return a.threads > 0 ? a.threads : kThreads; }

uint32_t apply_max_ctas(int num_sms, int blocks_per_sm) {
    const uint32_t g = (uint32_t)num_sms * (uint32_t)(blocks_per_sm > 0 ? blocks_per_sm : 8);
    return g < kApplyCluster ? kApplyCluster : g;
}

cudaError_t launch_apply(const DevInterner &I, const ApplyArgs &a, int mode, bool check_depths, bool clear_follows,
                         int num_sms, cudaStream_t s,
                         void (*levels_begin)(void *), void *levels_ctx) {
    const int bt = apply_threads_of(a);
    const uint64_t items = a.n_records > a.n_items ? a.n_records : a.n_items;
    const uint64_t cap = (uint64_t)num_sms * (uint64_t)(a.blocks_per_sm > 0 ? a.blocks_per_sm : 8);
    uint64_t g = (items + bt - 1) / bt;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    if (mode == 0) {
        count_launches(1);
        cudaError_t e = launch_pdl(apply_plan_kernel, dim3((unsigned)g), dim3(bt), 0, s, I, a, check_depths ? 1 : 0);
        if (e != cudaSuccess) return e;
    }
    count_launches(1);
    cudaError_t e = launch_pdl(apply_bottom_kernel, dim3((unsigned)g), dim3(bt), leaf_refs_smem(I), s, I, a, mode);
    if (levels_begin) (*levels_begin)(levels_ctx);
    for (int step = 1; step <= a.max_depth - 1 && a.n_records && e == cudaSuccess; ++step) {
        uint64_t gp = ((uint64_t)a.p_cap[step] + bt - 1) / bt;
        if (gp > cap) gp = cap;
        count_launches(1);
        e = launch_pdl(apply_parents_kernel, dim3((unsigned)gp), dim3(bt), leaf_refs_smem(I), s, I, a, mode, step, clear_follows ? 1 : 0);
    }
    return e;
}

cudaError_t launch_expand_items(const uint32_t *first, uint32_t n, uint32_t *rec_item, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    count_launches(1);
    expand_items_kernel<<<n < 65535u ? n : 65535u, kThreads, 0, s>>>(first, n, rec_item);
    return cudaGetLastError();
}

// Largest apply that runs as one cluster, a record a thread. Cluster against grid, an apply: 338 against 367 us for
// 476 records of a tree of depth 9, 390 against 406 for 3847, 493 against 421 for 7851; of chunks of depth 6 179
// against 206 for 981, 256 against 230 for 6780.
constexpr uint64_t kClusterRecords = 4096;

// The whole apply sequence in one launch: a small apply as one cluster, whose barrier is in hardware; else
// as many CTAs as can be resident at once (the grid barrier needs every CTA running).
cudaError_t launch_apply_single(const DevInterner &I, const ApplyArgs &a, bool check_depths, bool clear_pass,
                                uint32_t *frontier_a, uint32_t *frontier_b, int rounds, int num_sms, cudaStream_t s) {
    const size_t smem = std::max(leaf_refs_smem(I), release_smem(I.vbits));
    const uint64_t items = a.n_records > a.n_items ? a.n_records : a.n_items;
    int cd = check_depths ? 1 : 0, cp = clear_pass ? 1 : 0;
    if (items <= kClusterRecords) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kApplyCluster);
        cfg.blockDim = dim3(512);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kApplyCluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        count_launches(1);
        return cudaLaunchKernelEx(&cfg, apply_cluster_kernel, I, a, cd, cp, frontier_a, frontier_b, rounds);
    }
    const int bt = apply_threads_of(a);
    static int per_sm_cache[2][17] = {};  // [vbits == 16][threads / 32]
    int &per_sm = per_sm_cache[I.vbits == 16][bt / 32];
    if (per_sm == 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, apply_grid_kernel, bt, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
    }
    int want = a.blocks_per_sm > 0 ? a.blocks_per_sm : per_sm;
    if (want > per_sm) want = per_sm;
    // a small apply runs on as few CTAs as its records fill, no fewer than a quarter of the SMs: every
    // grid barrier costs one arrival per CTA
    uint64_t grid = (uint64_t)num_sms * want;
    const uint64_t fill = (items + bt - 1) / bt;
    const uint64_t floor_ctas = (uint64_t)(num_sms + 3) / 4;
    if (fill < grid) grid = fill > floor_ctas ? fill : floor_ctas;
    DevInterner Ic = I;
    ApplyArgs ac = a;
    void *args[] = {&Ic, &ac, &cd, &cp, &frontier_a, &frontier_b, &rounds};
    count_launches(1);
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(apply_grid_kernel), dim3((unsigned)grid), dim3(bt), args,
                                       smem, s);
}

}  // namespace vxg
