// Batched reads, releases, single-voxel edits and table maintenance.
//
//   get_many      VoxTree::get -> get_at_depth (voxtree.rs:145-159, utils/common.rs:122-156), one
//                 thread per query descending at most d levels through the L2-resident node array;
//                 large batches start from a table of the nodes some levels below every root.
//   release       dec_ref_recursive (interner/mod.rs:419-534) for many roots at once, breadth
//                 first: a round decrements the children of the nodes that died in the previous
//                 round; a child whose count reaches zero dies in the next round. Dead nodes leave
//                 their table, are cleared, get a new generation and go on the free list
//                 (recycle, interner/mod.rs:566-625). All rounds in one cooperative launch.
//   set / fill    VoxTree::set (voxtree.rs:163-260, 393-706) and fill/clear (voxtree.rs:264-292)
//                 by one CTA with the reference's own refcount order (hit: give back the children's
//                 references, interner/mod.rs:767-772), its LIFO free list and its 32768-entry
//                 release queue (P3 lifts the limit); one thread walks the path.
//   set many      many VoxTree::set calls at once, each tree's (or octant's) in call order.
//   to_dense      to_vec, a thread per quad; occupancy masks, a CTA per builder; serialisation.
//   rehash        rebuilds the branch table from the live nodes once tombstones accumulate.
#include <algorithm>
#include <type_traits>

#include "vx_launch.h"

namespace vxg {
namespace {

constexpr int kThreads = 256;

// The child of branch `node` in slot k, read through the read-only path; no load when the mask says EMPTY.
__device__ __forceinline__ uint64_t get_child(const DevInterner &I, uint64_t node, uint32_t k) {
    if (!((id_mask(node) >> k) & 1u)) return EMPTY_ID;
    return __ldg(reinterpret_cast<const unsigned long long *>(I.children) + 8ull * id_index(node) + k);
}

// Large batches of gets start from a table of the nodes k levels below every root: one load instead of k
// dependent ones. Tree t's entries are at t << 3k, by (y, z, x) of the node. In a tree of d <= k levels they are the
// nodes of depth d - 1: a leaf met above depth d is a voxel whatever its value, one at depth d only when that is not
// the default, and an entry does not say where its leaf was met.
__device__ __forceinline__ int get_levels(int d, int k) { return d > k ? k : (d > 0 ? d - 1 : 0); }

__device__ __forceinline__ uint32_t get_entry(uint32_t x, uint32_t y, uint32_t z, int d, int k) {
    return ((y >> (d - k)) << (2 * k)) | ((z >> (d - k)) << k) | (x >> (d - k));
}

__global__ void __launch_bounds__(kThreads) get_table_kernel(DevInterner I, uint32_t n_trees, int k, uint64_t *table) {
    const uint64_t n = (uint64_t)n_trees << (3 * k);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = (uint32_t)(i >> (3 * k)), e = (uint32_t)(i & ((1ull << (3 * k)) - 1ull));
        const int d = I.depths[t];
        if (d == TREE_UNUSED) continue;
        const int kt = get_levels(d, k);
        if (e >> (3 * kt)) continue;
        const uint32_t m = (1u << kt) - 1u, x = e & m, z = (e >> kt) & m, y = e >> (2 * kt);
        uint64_t node = I.roots[t];
        for (int s = kt - 1; s >= 0 && node != EMPTY_ID && id_is_branch(node); --s)
            node = get_child(I, node, ((x >> s) & 1u) | (((y >> s) & 1u) << 1) | (((z >> s) & 1u) << 2));
        table[i] = node;
    }
}

// One query a thread. (Two, four and eight chains of loads a thread, with 16-byte loads of the inputs, were
// slower at every size: 4 M gets on 4096 chunks 46 us with one, 49, 51 and 71 us.)
template <class T, bool TABLE>
__global__ void __launch_bounds__(kThreads) get_kernel(DevInterner I, uint64_t n, const uint32_t *trees,
                                                      const int32_t *xyz, uint8_t *found, T *values,
                                                      const uint64_t *table, int k, uint32_t n_trees) {
    if (TABLE) pdl_wait();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    bool oob = false, bad = false;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
        const uint32_t t = __ldg(trees + q);
        const uint32_t x = __ldg(xyz + 3 * q), y = __ldg(xyz + 3 * q + 1), z = __ldg(xyz + 3 * q + 2);
        const int d = t < I.tree_cap ? I.depths[t] : TREE_UNUSED;
        const uint32_t side = d == TREE_UNUSED ? 0u : 1u << d;
        const bool in = x < side && y < side && z < side;
        bad = bad || d == TREE_UNUSED;
        oob = oob || (d != TREE_UNUSED && !in);
        uint64_t node = EMPTY_ID;
        int shift = -1;  // of the child slot's coordinate bits, -1 at depth d
        if (in) {
            shift = d - 1;
            if (TABLE && t < n_trees) {  // (handles past the known ones: t < tree_cap)
                const int kt = get_levels(d, k);
                node = __ldg((const unsigned long long *)table + ((uint64_t)t << (3 * k)) + get_entry(x, y, z, d, kt));
                shift -= kt;
            } else {
                node = I.roots[t];
            }
        }
        for (; shift >= 0 && node != EMPTY_ID && id_is_branch(node); --shift)
            node = get_child(I, node, ((x >> shift) & 1) | (((y >> shift) & 1) << 1) | (((z >> shift) & 1) << 2));
        const uint32_t val = node != EMPTY_ID ? (uint32_t)__ldg(reinterpret_cast<const T *>(I.values) + id_index(node)) : 0u;
        found[q] = node != EMPTY_ID && (val != 0 || shift >= 0);  // at depth d a default value is no voxel
        values[q] = (T)val;
    }
    if (oob) set_error(I, ERR_OOB, 50);
    if (bad) set_error(I, ERR_INVALID, 51);
}

// ---- release (bodies in vx_device.cuh, shared with the single-launch apply) ------------------------
// The listed roots and then rounds until no node dies, one cooperative launch with a grid barrier after each
// (a launch per round, empty ones too, took 18 us a round on the few hundred nodes of a served wave).
// kReleaseCtas an SM, all resident, as the barrier needs: the bounds hold the registers to it, and release_smem is at
// most 32 KB.
constexpr int kReleaseCtas = 2;
__global__ void __launch_bounds__(kThreads, kReleaseCtas) release_kernel(DevInterner I, const uint64_t *list, uint32_t *frontier_a,
                                                           uint32_t *frontier_b, int rounds, int may_wait) {
    extern __shared__ uint32_t release_mem[];
    if (may_wait && *(volatile unsigned long long *)&I.ctr->scratch[SC_DEFER]) return;  // the list waits for the next release
    const uint64_t cta_base = (uint64_t)blockIdx.x * blockDim.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const bool t0 = cta_base + threadIdx.x == 0;
    DevCounters *ctr = I.ctr;
    GridBarrier bar(I);
    if (!bar.usable()) return;
    const LeafDrops D = leaf_drops_init(I, release_mem);
    // the counts are zero between launches: the rounds clear them, and the last one read is empty
    if (t0) ctr->scratch[SC_FREE_BASE] = ctr->free_count;
    release_roots_range(I, list, frontier_a, &ctr->rel_count[0], cta_base, stride);
    if (!bar.sync()) return;
    uint32_t *fr[2] = {frontier_a, frontier_b};
    uint64_t free_base = *(volatile unsigned long long *)&ctr->scratch[SC_FREE_BASE];
    int r = 0;
    for (; r < rounds; ++r) {
        const uint64_t n = *(volatile unsigned long long *)&ctr->rel_count[r % 3];
        if (n == 0) break;  // the same answer in every CTA
        if (t0) ctr->rel_count[(r + 2) % 3] = 0;
        release_round_range(I, D, fr[r & 1], fr[(r + 1) & 1], n, free_base, &ctr->rel_count[(r + 1) % 3], cta_base, stride);
        free_base += n;
        if (!bar.sync()) return;
    }
    if (t0) {  // set r % 3 was read by every CTA before its last barrier, or is the empty one
        ctr->rel_count[(r + 1) % 3] = 0;
        ctr->rel_count[(r + 2) % 3] = 0;
        if (r == rounds) ctr->rel_count[r % 3] = 0;
    }
    bar.leave();
}

// The answer of a one-tree call, in pinned host memory: the kernel writes it there itself, so that the call
// is one launch and one wait (a copy of the status and one of the counters took 8 us of a 29 us set, the
// argument and result copies of a get 25 of 38).
__device__ __forceinline__ void reply(const DevInterner &I, HostReply *r, int status, uint32_t value) {
    r->status = status;
    r->value = value;
    r->error = *(volatile unsigned int *)&I.ctr->error;
    r->tombstones = *(volatile unsigned long long *)&I.ctr->tombstones;
}

// VoxTree::get of one voxel inside the tree (voxtree.rs:145-159). status: found.
__global__ void tree_get_kernel(DevInterner I, uint32_t tree, uint32_t x, uint32_t y, uint32_t z, HostReply *r) {
    int shift = (int)I.depths[tree] - 1;
    uint64_t node = I.roots[tree];
    for (; shift >= 0 && node != EMPTY_ID && id_is_branch(node); --shift)
        node = get_child(I, node, ((x >> shift) & 1) | (((y >> shift) & 1) << 1) | (((z >> shift) & 1) << 2));
    const uint32_t val = node != EMPTY_ID ? node_value(I, id_index(node)) : 0u;
    reply(I, r, node != EMPTY_ID && (val != 0 || shift >= 0), val);
}

// ---- single-thread reference-order operations ---------------------------------------------------
struct Seq {
    DevInterner I;
    uint64_t *queue;
    uint64_t queue_cap;
    bool ok;
};

__device__ uint32_t seq_alloc(Seq &S) {
    DevCounters *c = S.I.ctr;
    if (c->free_count > 0) {
        c->free_count -= 1;
        c->created += 1;
        return S.I.free_list[c->free_count];
    }
    if (c->next_index >= S.I.capacity) {
        set_error(S.I, ERR_OOM, 70);
        S.ok = false;
        return NO_NODE;
    }
    c->created += 1;
    return (uint32_t)(c->next_index++);
}

__device__ void seq_recycle(Seq &S, uint32_t idx) {
    const uint64_t id = S.I.ids[idx];
    recycle_node(S.I, idx, id, S.I.hash[idx], S.I.generation[idx], S.I.ctr->free_count);
    S.I.ctr->free_count += 1;
    if (id_is_branch(id)) S.I.ctr->tombstones += 1;
}

__device__ bool seq_valid(Seq &S, uint64_t id) {
    const uint32_t i = id_index(id);
    return i < S.I.capacity && S.I.generation[i] == id_generation(id);
}

__device__ void seq_dec(Seq &S, uint64_t id) {  // dec_ref (interner/mod.rs:260-296)
    const uint32_t i = id_index(id);
    if (S.I.refcount[i] == 0) {
        set_error(S.I, ERR_REF_UB, 71);
        S.ok = false;
        return;
    }
    S.I.refcount[i] -= 1;
    if (S.I.refcount[i] == 0) seq_recycle(S, i);
}

// get_or_create_leaf (interner/mod.rs:627-710)
__device__ uint64_t seq_leaf(Seq &S, uint32_t v) {
    const uint64_t s = ld_volatile(S.I.leaf_table + v);  // a release before it works on L2
    if (s > LEAF_BUSY) {
        atomicAdd(S.I.refcount + id_index(s), 1u);
        return s;
    }
    const uint32_t idx = seq_alloc(S);
    if (idx == NO_NODE) return INVALID_ID;
    const uint64_t id = make_leaf_id(idx, S.I.generation[idx]);
    set_node_value(S.I, idx, v);
    S.I.hash[idx] = 0;
    S.I.ids[idx] = id;
    S.I.refcount[idx] = 1;
    S.I.leaf_table[v] = id;
    return id;
}

// get_or_create_branch (interner/mod.rs:712-829)
__device__ uint64_t seq_branch(Seq &S, const uint64_t c[8], uint32_t types, uint32_t mask) {
    const DevInterner &I = S.I;
    const uint64_t h = branch_fingerprint(c, (types << 8) | mask);
    const uint32_t tag = slot_tag(h);
    uint64_t pos = h & I.table_mask, tomb = ~0ull;  // the first tombstone met takes a new key
    for (uint32_t p = 0; p <= I.max_probes; ++p, pos = (pos + 1) & I.table_mask) {
        const uint64_t s = I.table[pos];
        if (s == SLOT_TOMB && tomb == ~0ull) tomb = pos;
        if (s == SLOT_EMPTY) {
            const uint32_t idx = seq_alloc(S);
            if (idx == NO_NODE) return INVALID_ID;
            if (tomb != ~0ull) {
                pos = tomb;
                I.ctr->tombstones -= 1;
            }
            uint32_t cv[8];
            for (int k = 0; k < 8; ++k) cv[k] = node_value(I, id_index(c[k]));
            const uint64_t id = write_branch(I, idx, c, types, mask, h, calc_average8(cv));
            I.refcount[idx] = 1;
            I.table[pos] = make_slot(tag, idx);
            return id;
        }
        if ((uint32_t)(s >> 32) == tag && s != SLOT_TOMB && key_equal(I, (uint32_t)s, c, types, mask)) {
            const uint64_t existing = I.ids[(uint32_t)s];
            for (int k = 0; k < 8; ++k)
                if (c[k] != EMPTY_ID) seq_dec(S, c[k]);
            I.refcount[(uint32_t)s] += 1;
            return existing;
        }
    }
    set_error(I, ERR_TABLE_FULL, 72);
    S.ok = false;
    return INVALID_ID;
}

// dec_ref_recursive (interner/mod.rs:419-534) with its fixed queue (grown under P3), by one CTA: a step's
// queue entries at a time, 8 threads each (one per child), with the queue, the counts and
// the order of the free list as the one-by-one loop leaves them. A child whose references all come from
// this step's entries dies and is queued where its last reference stands in the order of (entry, child);
// the occurrences of a dying child find that place through a small shared table. Entries of one step do
// not name each other (a queued node has lost every reference), and counts that say otherwise end the
// call as the underflow they are.
// Bound by the latency of a step's dependent loads (count and children, the children's counts, the table
// slot), about 2 us: clearing an edited 32^3 chunk took 2030 us in one thread, 108 us in steps of 32 entries. While
// more than 32 entries wait a step takes 128 (a CTA of 1024): 76 us against 110 for 4000 edited voxels of 32^3, 242
// against 467 for 20000 of 64^3; a few nodes are released by 256 threads as before (37 us, 45 when all 1024 took part).
constexpr int kSetThreads = 256;   // releases of a replaced path: narrow steps only
constexpr int kFillThreads = 1024;  // releases of whole trees

template <int kCta>
struct SeqShared {
    static constexpr uint32_t kRing = 2 * kCta;  // queue entries also kept in shared memory, the newest ones
    static constexpr uint32_t kLast = 2 * kCta;  // slots of the table of dying children
    static constexpr int kHomeShift = kCta == 256 ? 23 : 21;
    static_assert(kLast == 1u << (32 - kHomeShift), "the table's hash fills it");
    uint64_t ring[kRing];
    uint32_t key[kLast], last[kLast];  // node index + 1; last place of it among (entry, child)
    uint32_t pushes[kCta / 32], deaths[kCta / 32];
    unsigned long long r, w, free_count;  // place and end of the queue; length of the free list
    int ok;
};

// Barrier of the kN threads that take part in a step.
template <int kN, int kCta>
__device__ __forceinline__ void seq_bar() {
    if (kN == kCta)
        __syncthreads();
    else
        asm volatile("bar.sync 1, %0;" ::"n"(kN) : "memory");
}

// Steps of kN / 8 entries by the CTA's first kN threads, until the queue is empty or its length asks for the
// other width. S.ok and the queue are the same in every thread.
template <int kN, int kCta>
__device__ void seq_steps(Seq &S, SeqShared<kCta> &sh) {
    const DevInterner &I = S.I;
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, e = tid >> 3, k = tid & 7u;
    const unsigned lt = (1u << lane) - 1u;
    for (uint64_t r = sh.r;;) {
        const uint64_t w = sh.w, fc = sh.free_count;
        if (r >= w || !sh.ok) break;
        if (kCta != kSetThreads && (w - r > kSetThreads / 8) != (kN == kCta)) break;
        const uint32_t m = w - r < kN / 8 ? (uint32_t)(w - r) : kN / 8;
        const bool have = e < m;
        uint64_t child = EMPTY_ID, node = 0, h = 0;
        uint32_t ref = 0, gen = 0, ci = 0;
        if (have) {
            const uint64_t at = r + e;
            ci = id_index(w - at <= sh.kRing ? sh.ring[at % sh.kRing] : __ldcg((const unsigned long long *)S.queue + at));
            ref = __ldcg(I.refcount + ci);
            child = ld_cg(I.children + 8ull * ci + k);
            if (k == 0) {
                node = ld_cg(I.ids + ci);
                h = ld_cg(I.hash + ci);
                gen = I.generation[ci];
            }
        }
        const bool dying = have && ref == 1;
        if (!dying) child = EMPTY_ID;
        const uint32_t cc = id_index(child);
        const unsigned rec = __ballot_sync(0xFFFFFFFFu, dying && k == 0);
        if (lane == 0) sh.deaths[warp] = __popc(rec);
        seq_bar<kN, kCta>();  // every record of this step has been read
        uint32_t gone = 0, first = 0;
#pragma unroll
        for (unsigned x = 0; x < kN / 32; ++x) {
            if (x < warp) first += sh.deaths[x];
            gone += sh.deaths[x];
        }
        // the children lose their references while the entries that died leave the store, in queue order
        uint32_t old = 0;
        if (child != EMPTY_ID) old = atomicSub(I.refcount + cc, 1u);
        bool bad = have && ref == 0;
        if (have && k == 0) {
            if (atomicSub(I.refcount + ci, 1u) != ref) bad = true;  // the same node twice in one step
            if (dying) recycle_node(I, ci, node, h, gen, fc + first + __popc(rec & lt));
        }
        if (child != EMPTY_ID && old == 0) {
            atomicAdd(I.refcount + cc, 1u);
            bad = true;
        }
        if (bad) {
            set_error(I, ERR_REF_UB, 73);
            sh.ok = 0;
        }
        const unsigned tomb = __ballot_sync(0xFFFFFFFFu, dying && k == 0 && id_is_branch(node));
        if (lane == 0 && tomb) atomicAdd(&I.ctr->tombstones, (unsigned long long)__popc(tomb));
        const uint32_t home = (cc * 0x9E3779B1u) >> sh.kHomeShift;
        if (child != EMPTY_ID && old == 1)  // the last reference: the child dies
            for (uint32_t slot = home; atomicCAS(sh.key + slot, 0u, cc + 1u) != 0u;) slot = (slot + 1) & (sh.kLast - 1u);
        seq_bar<kN, kCta>();
        // the occurrences of each dying child find the last place of it
        uint32_t slot = home;
        bool dead = false;
        if (child != EMPTY_ID)
            for (;; slot = (slot + 1) & (sh.kLast - 1u)) {  // half of the slots stay free
                const uint32_t t = *(volatile uint32_t *)(sh.key + slot);
                dead = t == cc + 1u;
                if (dead || t == 0) break;
            }
        if (dead) atomicMax(sh.last + slot, tid);
        seq_bar<kN, kCta>();
        const bool push = dead && sh.last[slot] == tid;
        const unsigned b = __ballot_sync(0xFFFFFFFFu, push);
        if (lane == 0) sh.pushes[warp] = __popc(b);
        seq_bar<kN, kCta>();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (unsigned x = 0; x < kN / 32; ++x) {
            if (x < warp) before += sh.pushes[x];
            all += sh.pushes[x];
        }
        const bool full = w + all > S.queue_cap;
        if (push && !full) {
            const uint64_t at = w + before + __popc(b & lt);
            sh.ring[at % sh.kRing] = child;
            S.queue[at] = child;
            I.refcount[cc] = 1;  // its queue entry takes the last one
        }
        if (dead) {  // the shared table is empty again for the next step
            sh.key[slot] = 0;
            sh.last[slot] = 0;
        }
        if (tid == 0) {
            if (full) {
                set_error(I, ERR_REF_UB, 74);  // release queue overflow (interner/mod.rs:509-513)
                sh.ok = 0;
            }
            sh.free_count = fc + gone;
            sh.w = w + all;
        }
        r += m;
        if (tid == 0) sh.r = r;
        seq_bar<kN, kCta>();
    }
}

// The whole CTA calls it.
template <int kCta>
__device__ void seq_release(Seq &S, SeqShared<kCta> &sh, uint64_t root) {
    const unsigned tid = threadIdx.x;
    for (uint32_t s = tid; s < sh.kLast; s += kCta) sh.key[s] = 0, sh.last[s] = 0;
    if (tid == 0) {
        sh.ring[0] = root;
        sh.r = 0;
        sh.w = 1;
        sh.free_count = S.I.ctr->free_count;
        sh.ok = 1;
    }
    __syncthreads();
    for (;;) {
        if (tid < kSetThreads) seq_steps<kSetThreads, kCta>(S, sh);
        __syncthreads();
        if (kCta == kSetThreads || sh.r >= sh.w || !sh.ok) break;
        seq_steps<kCta, kCta>(S, sh);
        __syncthreads();  // every thread has seen the end of its steps before the next ones move it
    }
    if (tid == 0) S.I.ctr->free_count = sh.free_count;
    S.ok = sh.ok != 0;
    __syncthreads();
}

__device__ __forceinline__ uint32_t cidx(int32_t x, int32_t y, int32_t z, int cur, int max) {
    const int sh = max - cur - 1;
    return ((x >> sh) & 1) | (((y >> sh) & 1) << 1) | (((z >> sh) & 1) << 2);
}

// set_at_depth_iterative (voxtree.rs:393-540)
__device__ uint64_t seq_set(Seq &S, uint64_t root, int32_t x, int32_t y, int32_t z, int d, uint32_t voxel) {
    const DevInterner &I = S.I;
    uint64_t st_node[11], st_leaf[11];
    uint32_t st_idx[11];
    uint64_t cur = root, leaf = EMPTY_ID;
    int depth = 0;
    while (depth < d) {
        const uint32_t index = cidx(x, y, z, depth, d);
        if (id_is_branch(cur)) {
            st_node[depth] = cur;
            st_leaf[depth] = leaf;
            st_idx[depth] = index;
            cur = I.children[8ull * id_index(cur) + index];
        } else {
            if (node_value(I, id_index(cur)) == voxel) return INVALID_ID;
            leaf = cur;
            cur = EMPTY_ID;
            st_node[depth] = cur;
            st_leaf[depth] = leaf;
            st_idx[depth] = index;
        }
        ++depth;
    }
    if (id_is_leaf(cur) && node_value(I, id_index(cur)) == voxel) return INVALID_ID;
    cur = seq_leaf(S, voxel);
    while (depth > 0 && S.ok) {
        --depth;
        const uint64_t pn = st_node[depth], pl = st_leaf[depth];
        const uint32_t pi = st_idx[depth];
        if (pn != EMPTY_ID) {
            const uint32_t types = id_types(pn) | ((id_is_leaf(cur) ? 1u : 0u) << pi);
            uint64_t br[8];
            for (int k = 0; k < 8; ++k) br[k] = I.children[8ull * id_index(pn) + k];
            br[pi] = cur;
            bool same = types == 0xFF;
            for (int k = 0; k < 8; ++k) same = same && br[k] == cur;
            if (!same) {
                const uint32_t mask = id_mask(pn) | (1u << pi);
                for (int k = 0; k < 8; ++k)
                    if (k != (int)pi && br[k] != EMPTY_ID) I.refcount[id_index(br[k])] += 1;
                cur = seq_branch(S, br, types, mask);
            }
        } else if (pl == EMPTY_ID) {
            uint64_t ch[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            ch[pi] = cur;
            cur = seq_branch(S, ch, (id_is_leaf(cur) ? 1u : 0u) << pi, 1u << pi);
        } else {
            uint64_t ch[8];
            for (int k = 0; k < 8; ++k) ch[k] = pl;
            I.refcount[id_index(pl)] += 7;
            ch[pi] = cur;
            const uint32_t types = ((~(1u << pi)) | ((id_is_leaf(cur) ? 1u : 0u) << pi)) & 0xFFu;
            cur = seq_branch(S, ch, types, 0xFF);
        }
    }
    return cur;
}

// remove_at_depth / _branch / _leaf (voxtree.rs:542-706), unrolled into a descent and an ascent.
__device__ uint64_t seq_remove(Seq &S, uint64_t root, int32_t x, int32_t y, int32_t z, int d) {
    const DevInterner &I = S.I;
    uint64_t frames[11];
    int depth = 0;
    uint64_t node = root;
    uint64_t result;
    while (true) {
        if (!seq_valid(S, node)) {
            set_error(I, ERR_REF_PANIC, 75);
            S.ok = false;
            return INVALID_ID;
        }
        if (id_is_branch(node)) {
            if (!(depth < d)) {
                set_error(I, ERR_REF_PANIC, 76);  // "Branch node at max depth"
                S.ok = false;
                return INVALID_ID;
            }
            const uint32_t index = cidx(x, y, z, depth, d);
            if (!((id_mask(node) >> index) & 1)) return INVALID_ID;
            frames[depth] = node;
            node = I.children[8ull * id_index(node) + index];
            ++depth;
            continue;
        }
        // remove_at_depth_leaf from `depth` down to d, built bottom-up
        result = EMPTY_ID;
        for (int k = d - 1; k >= depth && S.ok; --k) {
            const uint32_t index = cidx(x, y, z, k, d);
            uint64_t ch[8];
            for (int j = 0; j < 8; ++j) ch[j] = node;
            ch[index] = result;
            const bool lf = id_is_leaf(result), em = result == EMPTY_ID;
            const uint32_t types = ((~(1u << index)) | ((lf ? 1u : 0u) << index)) & 0xFFu;
            const uint32_t mask = ((~(1u << index)) | ((!em ? 1u : 0u) << index)) & 0xFFu;
            I.refcount[id_index(node)] += 7;
            result = seq_branch(S, ch, types, mask);
        }
        break;
    }
    // ascend through the branch frames (remove_at_depth_branch)
    while (depth > 0 && S.ok) {
        --depth;
        const uint64_t pn = frames[depth];
        const uint32_t index = cidx(x, y, z, depth, d);
        const bool empty = result == EMPTY_ID;
        const uint32_t mask = empty ? (id_mask(pn) & ~(1u << index)) : id_mask(pn);
        if (mask == 0) {
            result = EMPTY_ID;
            continue;
        }
        if (!id_is_branch(result)) {
            set_error(I, ERR_REF_PANIC, 77);  // "Removing voxel should never produce a leaf node"
            S.ok = false;
            return INVALID_ID;
        }
        const uint32_t types = id_types(pn) & ~(1u << index);
        uint64_t br[8];
        for (int k = 0; k < 8; ++k) br[k] = I.children[8ull * id_index(pn) + k];
        br[index] = result;
        for (int k = 0; k < 8; ++k)
            if (k != (int)index && br[k] != EMPTY_ID) I.refcount[id_index(br[k])] += 1;
        result = seq_branch(S, br, types, mask);
    }
    return result;
}

// VoxTree::set (voxtree.rs:163-260). status: 0 unchanged, 1 changed, -1 error. Thread 0 runs the set, the
// CTA the release of the replaced root.
__global__ void __launch_bounds__(kSetThreads) tree_set_kernel(DevInterner I, uint32_t tree, int32_t x, int32_t y, int32_t z,
                                                               uint32_t v, uint64_t *queue, uint64_t queue_cap, HostReply *r) {
    __shared__ SeqShared<kSetThreads> sh;
    __shared__ uint64_t new_root;
    __shared__ int result;  // 0 unchanged, 1 to be installed, -1 error
    Seq S{I, queue, queue_cap, true};
    const uint64_t root = I.roots[tree];
    if (threadIdx.x == 0) {
        const int d = I.depths[tree];
        result = 0;
        if (root != EMPTY_ID || v != 0) {
            const uint64_t nw = v != 0 ? seq_set(S, root, x, y, z, d, v) : seq_remove(S, root, x, y, z, d);
            new_root = nw;
            if (!S.ok) {
                result = -1;
            } else if (nw != INVALID_ID) {
                result = 1;
                if (root != EMPTY_ID && nw == root) {
                    set_error(I, ERR_REF_PANIC, 78);
                    result = -1;
                }
            }
        }
    }
    __syncthreads();
    if (result == 1 && root != EMPTY_ID) seq_release(S, sh, root);
    if (threadIdx.x == 0) {
        if (result == 1 && S.ok) I.roots[tree] = new_root;
        reply(I, r, result == 1 && !S.ok ? -1 : result, 0);
    }
}

// ---- many VoxTree::set calls at once (vx_trees_set_many) ------------------------------------------
// The calls of one tree run in call order, one warp per tree (or per octant of it) and trees in parallel. Each call is the
// reference's set_at_depth_iterative / remove_at_depth (voxtree.rs:393-706) on the tree's current
// root, so every node it creates, including the stale types bits of the set path (the old parent's
// types ORed with the new child's leaf bit, voxtree.rs:513-514), is the node the reference creates.
// Refcounts are not touched during the calls and nothing is released: every node stays valid until the call
// ends, and a call that finds a node made by an earlier call gets the same node the reference would recreate.
// Afterwards the epoch refcount kernel counts one reference per child slot of every created node,
// the trees take their final roots (+1) and release their first ones, and created nodes that ended
// unreferenced (the intermediate roots and paths) are released, which leaves the refcounts the
// reference's per-call inc/dec bookkeeping gives.
//
// Bound by a call's chain of dependent round trips, so lane L of the warp is level L of the path. The descent
// leaves the path's rows of 8 children in the lanes; their values are loaded together. Going up, a level is
// looked up alone until the first new node: every node above it has a child that no key can name yet, so
// those are created together, a lane each, without comparing keys: one ticket range, and the slots, records
// and publications side by side. 8192 calls on 64 trees of depth 5: 1610 us, 3070 us when each level was
// looked up, allocated, written and published before the next.
struct Level {  // lane L's level of the path
    uint64_t c[8];   // children of the old node: a branch's, 8 copies of a leaf above it, or EMPTY
    uint32_t cv[8];  // their values
    uint64_t node, leaf;  // the branch at this level, or EMPTY and the leaf at or above it
    uint32_t pi;          // the path's child slot
};

// Slot of a new key in the branch table, claimed (BUSY): the first tombstone of its sequence, else its EMPTY
// slot. find: the key may be there or be created by another warp, whose node is then returned in *id;
// otherwise no slot can hold it. False (and an error) when the limits end the search.
__device__ __forceinline__ bool set_claim(const DevInterner &I, bool find, const uint64_t c[8], uint32_t types, uint32_t mask,
                                          uint64_t h, uint64_t *pos_out, uint64_t *id, bool *reused) {
    const uint32_t tag = slot_tag(h);
    uint64_t pos = h & I.table_mask;
    uint32_t probes = 0, tomb = 0, rounds = 0;
    for (;;) {
        uint64_t s = probe_sector(I, tag, pos, probes, tomb);
        if (s == SLOT_EMPTY) {
            if (tomb) {
                probes = tomb - 1;
                pos = (h + probes) & I.table_mask;
            }
            const uint64_t free_slot = tomb ? SLOT_TOMB : SLOT_EMPTY;
            const uint64_t prev = atomicCAS((unsigned long long *)(I.table + pos), free_slot, make_slot(tag, IDX_BUSY));
            if (prev == free_slot) {
                *pos_out = pos;
                *reused = tomb != 0;
                return true;
            }
            s = prev;
            tomb = 0;
        }
        if (find && (uint32_t)(s >> 32) == tag && s != SLOT_TOMB) {
            if ((uint32_t)s == IDX_BUSY) {  // being written by a warp that waits for nobody
                if (++rounds > I.round_limit) {
                    set_error(I, ERR_TIMEOUT, 2);
                    return false;
                }
                __nanosleep(32);
                continue;
            }
            if (key_equal(I, (uint32_t)s, c, types, mask, id)) return true;
        }
        if (s != SLOT_TOMB) {
            pos = (pos + 1) & I.table_mask;
            ++probes;
        }
        if (probes > I.max_probes) {
            set_error(I, ERR_TABLE_FULL, 1);
            return false;
        }
    }
}

// Types and mask of lane L's new node over child `cur` (set: voxtree.rs:500-539; remove: 559-705). Returns
// false when no node is made: all 8 children are the same leaf (the child stands for it), or none is left
// (*cur becomes EMPTY).
__device__ __forceinline__ bool set_level(const Level &P, bool remove, uint64_t *cur, uint32_t *types, uint32_t *mask) {
    const uint32_t bit = 1u << P.pi, lbit = id_is_leaf(*cur) ? bit : 0u;
    if (remove) {
        const uint32_t there = *cur == EMPTY_ID ? 0u : bit;
        if (P.node == EMPTY_ID) {  // the leaf above, split
            *types = 0xFFu & ~bit;
            *mask = (0xFFu & ~bit) | there;
            return true;
        }
        *types = id_types(P.node) & ~bit;
        *mask = *cur == EMPTY_ID ? id_mask(P.node) & ~bit : id_mask(P.node);
        if (*mask == 0) *cur = EMPTY_ID;
        return *mask != 0;
    }
    if (P.node != EMPTY_ID) {
        *types = id_types(P.node) | lbit;
        *mask = id_mask(P.node) | bit;
        bool same = *types == 0xFF;
#pragma unroll
        for (int k = 0; k < 8; ++k) same = same && ((uint32_t)k == P.pi || P.c[k] == *cur);
        return !same;
    }
    *types = P.leaf == EMPTY_ID ? lbit : (0xFFu & ~bit) | lbit;
    *mask = P.leaf == EMPTY_ID ? bit : 0xFFu;
    return true;
}

__device__ __forceinline__ void put_child(Level &P, uint64_t id, uint32_t value) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if ((uint32_t)k == P.pi) {
            P.c[k] = id;
            P.cv[k] = value;
        }
}

// One call by one warp: the new root, INVALID_ID when nothing changes; *ok is cleared on an error.
__device__ uint64_t warp_set(const DevInterner &I, unsigned long long fc, unsigned long long ni, uint64_t root, int32_t x,
                             int32_t y, int32_t z, int d, uint32_t voxel, bool *ok) {
    const unsigned lane = threadIdx.x & 31u;
    const bool remove = voxel == 0;
    constexpr unsigned kAll = 0xFFFFFFFFu;
    uint64_t leaf_id = voxel ? ld_volatile(I.leaf_table + voxel) : EMPTY_ID;  // beside the descent's loads
    Level P;
    P.node = P.leaf = EMPTY_ID;
    P.pi = (int)lane < d ? cidx(x, y, z, lane, d) : 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) P.c[k] = EMPTY_ID;
    uint64_t cur = root, above = EMPTY_ID;  // above: the leaf the path ran into
    for (int L = 0; L < d; ++L) {
        if (cur == EMPTY_ID) {
            if (remove) return INVALID_ID;
            break;
        }
        if (id_is_leaf(cur)) {
            above = cur;
            break;
        }
        if (remove && !__shfl_sync(kAll, (id_mask(cur) >> P.pi) & 1u, L)) return INVALID_ID;
        uint64_t next = EMPTY_ID;
        if ((int)lane == L) {
            P.node = cur;
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * id_index(cur));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ulonglong2 w = __ldcg(src + k);
                P.c[2 * k] = w.x;
                P.c[2 * k + 1] = w.y;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if ((uint32_t)k == P.pi) next = P.c[k];
        }
        cur = __shfl_sync(kAll, next, L);
    }
    if (remove && above == EMPTY_ID && id_is_branch(cur)) {  // at depth d
        set_error(I, ERR_REF_PANIC, 80);  // "Branch node at max depth"
        *ok = false;
        return INVALID_ID;
    }
    // the values of the rows, and whether the voxel has its value already
    const uint64_t met = above != EMPTY_ID ? above : cur;
    uint32_t met_value = 0;
    if (met != EMPTY_ID && id_is_leaf(met)) met_value = node_value_cg(I, id_index(met));
    if (P.node == EMPTY_ID && (int)lane < d) {
        P.leaf = above;
#pragma unroll
        for (int k = 0; k < 8; ++k) P.c[k] = above;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) P.cv[k] = (P.node != EMPTY_ID && P.c[k] != EMPTY_ID) ? node_value_cg(I, id_index(P.c[k])) : 0u;
    if (!remove && met != EMPTY_ID && id_is_leaf(met) && met_value == voxel) return INVALID_ID;
    if (P.leaf != EMPTY_ID) {
#pragma unroll
        for (int k = 0; k < 8; ++k) P.cv[k] = met_value;
    }
    if (voxel && leaf_id <= LEAF_BUSY) {
        bool created;
        leaf_id = lane == 0 ? intern_leaf(I, voxel, &created) : EMPTY_ID;
        leaf_id = __shfl_sync(kAll, leaf_id, 0);
        if (leaf_id == EMPTY_ID) {
            *ok = false;
            return INVALID_ID;
        }
    }
    // up to the first new node, a level at a time
    cur = leaf_id;
    uint32_t value = voxel;
    uint64_t pos = 0;
    bool reused = false;
    uint64_t h = 0;
    uint32_t types = 0, mask = 0, lod = 0;
    int L = d - 1;
    for (; L >= 0; --L) {
        int what = 0;  // 0: no node, 1: found, 2: claimed, 3: failed
        uint64_t id = EMPTY_ID;
        if ((int)lane == L) {
            id = cur;
            if (set_level(P, remove, &id, &types, &mask)) {
                put_child(P, id, value);
                lod = calc_average8(P.cv);
                h = branch_fingerprint(P.c, (types << 8) | mask);
                id = EMPTY_ID;
                what = set_claim(I, true, P.c, types, mask, h, &pos, &id, &reused) ? (id != EMPTY_ID ? 1 : 2) : 3;
            }
        }
        what = __shfl_sync(kAll, what, L);
        if (what == 3) {
            *ok = false;
            return INVALID_ID;
        }
        if (what == 2) break;
        cur = __shfl_sync(kAll, id, L);
        value = what == 0 ? (cur == EMPTY_ID ? 0u : value) : __shfl_sync(kAll, lod, L);
    }
    if (L < 0) return cur;
    // levels L .. 0 are new nodes: lane j <= L makes level j, tickets bottom up
    const bool mine = (int)lane <= L;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&I.ctr->alloc_count, (unsigned long long)(L + 1));
    // while the ticket is fetched: types and masks above level L, whose children are branches, and the values
    if ((int)lane < L) {
        uint64_t child = 2;  // some branch
        (void)set_level(P, remove, &child, &types, &mask);
    }
    for (int j = L - 1; j >= 0; --j) {
        const uint32_t below = __shfl_sync(kAll, lod, j + 1);
        if ((int)lane == j) {
            put_child(P, EMPTY_ID, below);
            lod = calc_average8(P.cv);
        }
    }
    base = __shfl_sync(kAll, base & kTicketMask, 0);
    const unsigned long long t = base + (unsigned long long)(L - (int)lane);
    const uint32_t idx = mine ? node_for_ticket(I, t, fc, ni) : 0u;
    if (__any_sync(kAll, mine && idx == NO_NODE)) {
        if ((int)lane == L) {
            set_error(I, ERR_OOM, 1);
            atomicExch((unsigned long long *)(I.table + pos), SLOT_TOMB);
        }
        *ok = false;
        return INVALID_ID;
    }
    const uint64_t id = mine ? make_branch_id(idx, slot_generation(I, idx, t >= fc), types, mask) : EMPTY_ID;
    const uint64_t child = __shfl_down_sync(kAll, id, 1);
    bool claimed = (int)lane == L, failed = false;
    if ((int)lane < L) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if ((uint32_t)k == P.pi) P.c[k] = child;
        h = branch_fingerprint(P.c, (types << 8) | mask);
        uint64_t other;
        claimed = set_claim(I, false, P.c, types, mask, h, &pos, &other, &reused);
        failed = !claimed;
    }
    failed = __any_sync(kAll, failed);
    if (mine && !failed) write_branch(I, idx, P.c, types, mask, h, lod, t >= fc);
    const unsigned re = __ballot_sync(kAll, mine && claimed && reused && !failed);
    if (lane == 0 && re) atomicAdd(&I.ctr->alloc_count, (unsigned long long)__popc(re) << kTicketBits);
    if (mine && claimed) publish_release((unsigned long long *)(I.table + pos), failed ? SLOT_TOMB : make_slot(slot_tag(h), idx));
    if (failed) {
        *ok = false;
        return INVALID_ID;
    }
    __syncwarp();  // the next call reads these records in other lanes
    return __shfl_sync(kAll, id, 0);
}

// Calls [begin[g], begin[g+1]) of group g's tree in call order, by one warp.
__device__ void set_calls_in_order(const DevInterner &I, const SetCalls &c, uint32_t g, unsigned long long fc,
                                   unsigned long long ni) {
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t tree = c.group_tree[g];
    const int d = I.depths[tree];
    uint64_t root = I.roots[tree];
    bool ok = true;
    const uint32_t first = c.begin[g], end = c.begin[g + 1];
    for (uint32_t k0 = first; k0 < end && ok; k0 += 32) {  // 32 calls' arguments at a time
        const uint32_t m = end - k0 < 32 ? end - k0 : 32;
        int32_t ax = 0, ay = 0, az = 0;
        uint32_t av = 0;
        if (lane < m) {
            ax = c.xyz[3 * (uint64_t)(k0 + lane)];
            ay = c.xyz[3 * (uint64_t)(k0 + lane) + 1];
            az = c.xyz[3 * (uint64_t)(k0 + lane) + 2];
            av = c.values[k0 + lane];
        }
        uint8_t changed = 0;  // of call k0 + lane
        uint32_t k = 0;
        for (; k < m; ++k) {
            const int32_t x = __shfl_sync(0xFFFFFFFFu, ax, k), y = __shfl_sync(0xFFFFFFFFu, ay, k),
                          z = __shfl_sync(0xFFFFFFFFu, az, k);
            const uint32_t v = __shfl_sync(0xFFFFFFFFu, av, k);
            if (root == EMPTY_ID && v == 0) continue;
            const uint64_t nw = warp_set(I, fc, ni, root, x, y, z, d, v, &ok);
            if (!ok) break;
            if (nw == INVALID_ID) continue;
            if (root != EMPTY_ID && nw == root) {  // assert_ne!(new_root_id, self.root_id)
                set_error(I, ERR_REF_PANIC, 82);
                ok = false;
                break;
            }
            root = nw;
            if (lane == k) changed = 1;
        }
        if (lane < k && c.changed) c.changed[c.order[k0 + lane]] = changed;
    }
    if (lane == 0) c.new_root[g] = root;
}

// One warp per tree.
__global__ void __launch_bounds__(32) trees_set_kernel(DevInterner I, const SetCalls c) {
    if (blockIdx.x == 0 && threadIdx.x == 0) I.ctr->scratch[SC_RELEASE] = 0;
    const unsigned long long fc = I.ctr->free_count, ni = I.ctr->next_index;  // fixed during the epoch
    for (uint32_t g = blockIdx.x; g < c.n_groups; g += gridDim.x) set_calls_in_order(I, c, g, fc, ni);
}

// The root of a tree over its 8 octants, as the calls move it one after the other (set_level at level 0).
struct RootState {
    uint64_t c[8];
    uint64_t whole;        // the leaf that the root is, or EMPTY, when it is no branch
    uint32_t types, mask;  // of the branch
    bool branch;

    // The call replaces octant o by id. False when the 8 octants collapse into one that is no leaf.
    __device__ bool apply(uint32_t o, uint64_t id, bool remove) {
        const uint32_t bit = 1u << o, lbit = id_is_leaf(id) ? bit : 0u;
        bool same = true;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if ((uint32_t)k == o) c[k] = id;
            same = same && c[k] == id;
        }
        if (branch) {
            if (remove) {
                types &= ~bit;
                if (id == EMPTY_ID) mask &= ~bit;
            } else {
                types |= lbit;
                mask |= bit;
                if (types == 0xFF && same) {
                    branch = false;
                    whole = id;
                    return id_is_leaf(id);
                }
            }
        } else {
            const bool leaf = whole != EMPTY_ID;  // (a call that changes an EMPTY tree sets)
            types = (leaf ? 0xFFu & ~bit : 0u) | (remove ? 0u : lbit);
            mask = (leaf ? 0xFFu & ~bit : 0u) | (id != EMPTY_ID ? bit : 0u);
            branch = true;
        }
        if (mask == 0) {
            branch = false;
            whole = EMPTY_ID;
        }
        return true;
    }
};

// Trees with many calls: a CTA per tree, a warp per octant of it. A call below one octant reads and makes no node
// of another, so the octants' calls run side by side, each octant's in order, and only the root is the work of
// them all: its state is replayed from the octants' ids in call order (a leaf's type bit stays set when a set
// splits it, and the root collapses into a leaf and splits again, as order has it), and its node made once. Where
// the one-by-one calls would end in an error, or 8 equal branches collapse, the calls are run again in order.
constexpr int kOctantThreads = 256;

__global__ void __launch_bounds__(kOctantThreads) trees_set_octants_kernel(DevInterner I, const SetCalls c) {
    __shared__ int redo;
    if (blockIdx.x == 0 && threadIdx.x == 0) I.ctr->scratch[SC_RELEASE] = 0;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const unsigned long long fc = I.ctr->free_count, ni = I.ctr->next_index;  // fixed during the epoch
    for (uint32_t g = blockIdx.x; g < c.n_groups; g += gridDim.x) {
        const uint32_t tree = c.group_tree[g];
        const int d = I.depths[tree];
        const uint64_t root = I.roots[tree];
        const uint32_t first = c.begin[g], end = c.begin[g + 1];
        if (threadIdx.x == 0) redo = d < 2;
        __syncthreads();
        if (d >= 2) {
            uint64_t octant = id_is_leaf(root) ? root : EMPTY_ID;
            if (root != EMPTY_ID && id_is_branch(root)) octant = ld_cg(I.children + 8ull * id_index(root) + warp);
            const int32_t low = (1 << (d - 1)) - 1;
            bool ok = true;
            for (uint32_t k0 = first; k0 < end && ok; k0 += 32) {
                const bool in = k0 + lane < end;
                int32_t ax = 0, ay = 0, az = 0;
                uint32_t av = 0, o = 8;
                if (in) {
                    ax = c.xyz[3 * (uint64_t)(k0 + lane)];
                    ay = c.xyz[3 * (uint64_t)(k0 + lane) + 1];
                    az = c.xyz[3 * (uint64_t)(k0 + lane) + 2];
                    av = c.values[k0 + lane];
                    o = cidx(ax, ay, az, 0, d);
                }
                uint64_t result = INVALID_ID;
                for (unsigned todo = __ballot_sync(kAll, o == warp); todo && ok; todo &= todo - 1) {
                    const int k = __ffs(todo) - 1;
                    const int32_t x = __shfl_sync(kAll, ax, k) & low, y = __shfl_sync(kAll, ay, k) & low,
                                  z = __shfl_sync(kAll, az, k) & low;
                    const uint32_t v = __shfl_sync(kAll, av, k);
                    if (octant == EMPTY_ID && v == 0) continue;
                    const uint64_t nw = warp_set(I, fc, ni, octant, x, y, z, d - 1, v, &ok);
                    if (!ok || nw == INVALID_ID) continue;
                    ok = nw != octant;
                    octant = nw;
                    if ((int)lane == k) result = nw;
                }
                if (o == warp) c.results[k0 + lane] = result;
            }
            if (!ok && lane == 0) redo = 1;
        }
        __syncthreads();
        if (warp == 0 && !redo) {
            RootState R;
            R.branch = root != EMPTY_ID && id_is_branch(root);
            R.whole = R.branch ? EMPTY_ID : root;
            R.types = id_types(root);
            R.mask = id_mask(root);
#pragma unroll
            for (int k = 0; k < 8; ++k) R.c[k] = R.branch ? ld_cg(I.children + 8ull * id_index(root) + k) : root;
            bool any = false, ok = true;
            for (uint32_t k0 = first; k0 < end; k0 += 32) {
                const bool in = k0 + lane < end;
                uint64_t result = INVALID_ID;
                uint32_t o = 0;
                bool remove = false;
                if (in) {
                    const uint64_t k = k0 + lane;
                    result = ld_cg(c.results + k);
                    o = cidx(c.xyz[3 * k], c.xyz[3 * k + 1], c.xyz[3 * k + 2], 0, d);
                    remove = c.values[k] == 0;
                    if (c.changed) c.changed[c.order[k]] = result != INVALID_ID;
                }
                for (unsigned todo = __ballot_sync(kAll, result != INVALID_ID); todo; todo &= todo - 1) {
                    const int k = __ffs(todo) - 1;
                    any = true;
                    ok = R.apply(__shfl_sync(kAll, o, k), __shfl_sync(kAll, result, k), __shfl_sync(kAll, (int)remove, k) != 0) && ok;
                }
            }
            uint64_t nw = root;
            if (any && ok) {
                nw = R.whole;
                if (R.branch) {
                    uint32_t cv[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) cv[k] = R.c[k] != EMPTY_ID ? node_value_cg(I, id_index(R.c[k])) : 0u;
                    bool created;
                    nw = warp_intern_branch(I, lane == 0, R.c, R.types, R.mask, calc_average8(cv), &created);
                    nw = __shfl_sync(kAll, nw, 0);
                    if (nw == EMPTY_ID) nw = root;  // (its error is recorded)
                }
            }
            if (lane == 0) {
                c.new_root[g] = nw;
                redo = !ok;
            }
            __syncwarp();
        }
        __syncthreads();
        if (warp == 0 && redo) set_calls_in_order(I, c, g, fc, ni);
        __syncthreads();
    }
}

// The trees take their final roots (one reference each) and list their first roots for release.
__global__ void __launch_bounds__(kThreads) trees_set_roots_kernel(DevInterner I, const SetCalls c, uint64_t *list) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < c.n_groups; g += gridDim.x * blockDim.x) {
        const uint32_t tree = c.group_tree[g];
        const uint64_t old = I.roots[tree], nw = c.new_root[g];
        if (nw == old) continue;
        I.roots[tree] = nw;
        if (nw != EMPTY_ID) atomicAdd(I.refcount + id_index(nw), 1u);
        if (old != EMPTY_ID) list[atomicAdd(&I.ctr->scratch[SC_RELEASE], 1ull)] = old;
    }
}

// Created nodes left without a reference are listed for release with a count of one. The created
// slots are free_list[free_count .. fc0) and [ni0, next_index) once the epoch is closed.
__global__ void __launch_bounds__(kThreads) trees_set_garbage_kernel(DevInterner I, unsigned long long fc0,
                                                                    unsigned long long ni0, uint64_t *list) {
    const unsigned long long fc = I.ctr->free_count, ni = I.ctr->next_index;
    const unsigned long long n_free = fc0 - fc, n = n_free + (ni - ni0);
    for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < n;
         t += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t idx = t < n_free ? I.free_list[fc + t] : (uint32_t)(ni0 + (t - n_free));
        const uint64_t id = I.ids[idx];
        if (id == EMPTY_ID || I.refcount[idx] != 0) continue;
        I.refcount[idx] = 1;
        list[atomicAdd(&I.ctr->scratch[SC_RELEASE], 1ull)] = id;
    }
}

// VoxTree::fill / clear (voxtree.rs:264-292). status: 1 if the tree was dirtied. One CTA.
__global__ void __launch_bounds__(kFillThreads) tree_fill_kernel(DevInterner I, uint32_t tree, uint32_t v, uint64_t *queue,
                                                                uint64_t queue_cap, HostReply *r) {
    __shared__ SeqShared<kFillThreads> sh;
    Seq S{I, queue, queue_cap, true};
    const uint64_t root = I.roots[tree];
    __syncthreads();
    if (root != EMPTY_ID) seq_release(S, sh, root);
    if (threadIdx.x != 0) return;
    int status = root != EMPTY_ID;
    if (S.ok && root != EMPTY_ID) I.roots[tree] = EMPTY_ID;
    if (S.ok && v != 0) {
        const uint64_t leaf = seq_leaf(S, v);
        if (S.ok) I.roots[tree] = leaf;
        status = 1;
    }
    reply(I, r, S.ok ? status : -1, 0);
}

// ---- maintenance -------------------------------------------------------------------------------
__global__ void rehash_kernel(DevInterner I) {
    const unsigned long long n = I.ctr->next_index;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x + 1; idx < n;
         idx += stride) {
        const uint64_t id = I.ids[idx];
        if (id == 0 || id_is_leaf(id)) continue;
        const uint64_t h = I.hash[idx];
        uint64_t pos = h & I.table_mask;
        const uint64_t slot = make_slot(slot_tag(h), (uint32_t)idx);
        bool placed = false;
        for (uint32_t p = 0; p <= I.max_probes; ++p, pos = (pos + 1) & I.table_mask)
            if (atomicCAS((unsigned long long *)(I.table + pos), SLOT_EMPTY, slot) == SLOT_EMPTY) {
                placed = true;
                break;
            }
        if (!placed) set_error(I, ERR_TABLE_FULL, 80);
    }
}

__global__ void rehash_done_kernel(DevInterner I) { I.ctr->tombstones = 0; }

// The interner back in its created state, by the slots that were handed out instead of the whole capacity
// (slots past them still are as created: node_for_ticket hands out each once). The branch table is cleared
// through its keys when they are few and nothing but live keys is in it: every branch clears the run of full
// slots from its home on. A run that another thread cleared in part is finished by that thread, so every
// key's slot is reached. Else the whole table is cleared. The last CTA writes the counters.
// About 60,000 nodes in a 64 MiB interner: 9 us; nine memsets over the capacity took 28 us and 36 us to queue.
__global__ void __launch_bounds__(kThreads) reset_kernel(DevInterner I) {
    const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const DevCounters *c = I.ctr;
    const unsigned long long open = c->alloc_count & kTicketMask;  // of an epoch that was not closed
    unsigned long long n = c->next_index + open;
    if (n > I.capacity) n = I.capacity;
    const uint64_t slots = I.table_mask + 1;
    const bool by_key = c->tombstones == 0 && c->error == 0 && open == 0 && n * 8 <= slots;
    for (uint64_t i = gt; i < n; i += stride) {
        const uint64_t id = I.ids[i];
        if (by_key && id != 0 && id_is_branch(id))
            for (uint64_t pos = I.hash[i] & I.table_mask; ld_volatile(I.table + pos) != SLOT_EMPTY; pos = (pos + 1) & I.table_mask)
                *(volatile uint64_t *)(I.table + pos) = SLOT_EMPTY;
        ulonglong2 *ch = reinterpret_cast<ulonglong2 *>(I.children + 8ull * i);
        ch[0] = ch[1] = ch[2] = ch[3] = make_ulonglong2(0ull, 0ull);
        set_node_value(I, (uint32_t)i, 0);
        I.refcount[i] = 0;
        I.generation[i] = 0;
        I.hash[i] = 0;
        I.ids[i] = 0;
    }
    if (!by_key) {
        ulonglong2 *t = reinterpret_cast<ulonglong2 *>(I.table);  // a power of two of slots; one slot: below
        for (uint64_t i = gt; i < slots / 2; i += stride) t[i] = make_ulonglong2(SLOT_EMPTY, SLOT_EMPTY);
        if (slots == 1 && gt == 0) I.table[0] = SLOT_EMPTY;
    }
    for (uint64_t i = gt; i < (1ull << I.vbits); i += stride) I.leaf_table[i] = 0;
    for (uint64_t i = gt; i < I.tree_cap; i += stride) I.roots[i] = 0;
    if (grid_last_cta(&I.ctr->scratch[SC_DONE])) {
        *I.ctr = DevCounters{};
        I.ctr->next_index = 1;
    }
}

__global__ void count_live_kernel(DevInterner I, unsigned long long *out2) {
    const unsigned long long n = I.ctr->next_index;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long br = 0, lf = 0;
    for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x + 1; idx < n;
         idx += stride) {
        const uint64_t id = I.ids[idx];
        if (id == 0) continue;
        if (id_is_leaf(id))
            ++lf;
        else
            ++br;
    }
    for (int o = 16; o > 0; o >>= 1) {
        br += __shfl_down_sync(0xFFFFFFFFu, br, o);
        lf += __shfl_down_sync(0xFFFFFFFFu, lf, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (br) atomicAdd(out2, br);
        if (lf) atomicAdd(out2 + 1, lf);
    }
}


// ---- to_vec: DAG -> dense grid (utils/common.rs:158-246) ----------------------------------------
// One thread per quad (4^3 voxels). The thread descends from its tree's root to the quad's node (d - 2
// levels; lanes of a warp share most of the path, so these loads are L1 hits); EMPTY or a leaf met on
// the way makes the quad uniform (EMPTY children are never visited by to_vec, leaving the default; a
// leaf fills its whole sub-cube). Otherwise the quad's 8 groups are resolved to voxels: EMPTY, a leaf's
// value, or the values of the nodes at depth d, as to_vec's else-branch does. The 16 rows of 4 voxels go
// straight from registers to the output.
// Nothing is staged: no shared memory, no CTA barrier, every quad independent; bound by instruction
// issue and the latency of the gathers (ncu: issue 59%, DRAM 17%). Quads of a cube of side 32 are
// numbered x first, then z, then y: a warp covers 8 x 4 quads of one y, so each of its stores writes
// whole 32-byte sectors (u8) and its lanes share nodes.
// 4096 dune chunks of 32^3 u8 (134 MB): 60 us, one 512^3 u8 cave tree: 78 us (132 and 180 us when a CTA
// expanded each 32^3 cube level by level in 68 KB of shared memory, with a barrier per level). Slower:
// four lanes resolving four quads together, 16 bytes of a node record each (77 and 118 us); exchanging
// rows between lanes for 16-byte stores (no gain).
constexpr int kDenseOutThreads = 256;

__device__ __forceinline__ uint64_t child_ro(const DevInterner &I, uint64_t id, uint32_t k) {
    return __ldg(reinterpret_cast<const unsigned long long *>(I.children) + 8ull * id_index(id) + k);
}

template <class T>
__device__ __forceinline__ uint32_t value_ro(const DevInterner &I, uint64_t id) {
    return __ldg(reinterpret_cast<const T *>(I.values) + id_index(id));
}

// The 8 voxels under a bottom group's node (or above it: an EMPTY or leaf ancestor), x fastest, then y,
// then z, as two bytes or 16-bit elements a word: w[y + 2z] = v(0, y, z) | v(1, y, z) << bits.
template <class T>
__device__ __forceinline__ void group_rows(const DevInterner &I, uint64_t g, uint32_t w[4]) {
    constexpr int B = 8 * sizeof(T);
    if (g == EMPTY_ID) {
#pragma unroll
        for (int r = 0; r < 4; ++r) w[r] = 0;
    } else if (id_is_leaf(g)) {
        const uint32_t v = value_ro<T>(I, g);
#pragma unroll
        for (int r = 0; r < 4; ++r) w[r] = v | (v << B);
    } else {
        const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * id_index(g));
        ulonglong2 c[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) c[r] = __ldg(src + r);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t lo = c[r].x ? value_ro<T>(I, c[r].x) : 0u, hi = c[r].y ? value_ro<T>(I, c[r].y) : 0u;
            w[r] = lo | (hi << B);
        }
    }
}

template <class T>
__global__ void __launch_bounds__(kDenseOutThreads) to_dense_kernel(DevInterner I, const uint32_t *trees, int d,
                                                                     uint64_t cube_begin, uint64_t n_cubes, T *out) {
    using Row = typename std::conditional<sizeof(T) == 1, uint32_t, uint2>::type;  // 4 voxels along x
    const int qb = (d < 5 ? d : 5) - 2;    // quads a cube has along an axis, log2
    const int kb = d - 2 - qb;             // cubes a tree has along an axis, log2
    const uint32_t qm = (1u << qb) - 1u, km = (1u << kb) - 1u;
    const uint64_t S = 1ull << d, S2 = S * S;
    const uint64_t total = n_cubes << (3 * qb);
    const uint64_t first_row = (cube_begin >> (2 * kb)) << (qb + 2);  // out starts at this y of the trees' stack
    bool bad = false;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t cube = cube_begin + (q >> (3 * qb));
        const uint32_t c = (uint32_t)cube, w = (uint32_t)q;
        const uint32_t X = ((c & km) << qb) | (w & qm);  // quad coordinates in the tree
        const uint32_t Z = (((c >> kb) & km) << qb) | ((w >> qb) & qm);
        const uint32_t Y = (((c >> (2 * kb)) & km) << qb) | ((w >> (2 * qb)) & qm);
        const uint64_t t_idx = cube >> (3 * kb);
        const uint32_t t = __ldg(trees + t_idx);
        uint64_t node = EMPTY_ID;
        if (t < I.tree_cap && I.depths[t] == d)
            node = I.roots[t];
        else
            bad = true;
        for (int sh = d - 3; sh >= 0 && node != EMPTY_ID && !id_is_leaf(node); --sh)
            node = child_ro(I, node, ((X >> sh) & 1) | (((Y >> sh) & 1) << 1) | (((Z >> sh) & 1) << 2));
        T *dst = out + ((t_idx << d) + 4 * Y - first_row) * S2 + 4 * Z * S + 4 * X;
        uint64_t g[8];
        const bool split = node != EMPTY_ID && !id_is_leaf(node);
        if (split) {
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * id_index(node));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ulonglong2 v = __ldg(src + k);
                g[2 * k] = v.x;
                g[2 * k + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) g[k] = node;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // the two groups along x at (gy, gz)
            const int gy = k & 1, gz = k >> 1;
            uint32_t a[4], b[4];
            group_rows<T>(I, g[2 * k], a);
            if (split) {
                group_rows<T>(I, g[2 * k + 1], b);
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r) b[r] = a[r];
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                Row *p = reinterpret_cast<Row *>(dst + (2 * gy + (r & 1)) * S2 + (2 * gz + (r >> 1)) * S);
                if constexpr (sizeof(T) == 1)
                    *p = a[r] | (b[r] << 16);
                else
                    *p = make_uint2(a[r], b[r]);
            }
        }
    }
    if (bad) set_error(I, ERR_INVALID, 52);
}

// Trees of depth 1: one thread per tree, 8 voxels.
template <class T>
__global__ void __launch_bounds__(kDenseOutThreads) to_dense_depth1_kernel(DevInterner I, const uint32_t *trees,
                                                                            uint64_t begin, uint64_t n, T *out) {
    bool bad = false;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = __ldg(trees + begin + i);
        uint64_t node = EMPTY_ID;
        if (t < I.tree_cap && I.depths[t] == 1)
            node = I.roots[t];
        else
            bad = true;
        uint32_t w[4];
        group_rows<T>(I, node, w);
#pragma unroll
        for (int r = 0; r < 4; ++r) {  // w[y + 2z] holds row (y, z); the grid is [y][z][x]
            T *row = out + 8 * i + 4 * (r & 1) + 2 * (r >> 1);
            row[0] = (T)w[r];
            row[1] = (T)(w[r] >> (8 * sizeof(T)));
        }
    }
    if (bad) set_error(I, ERR_INVALID, 52);
}
}  // namespace


// ---- occupancy masks for greedy meshing (utils/mesh.rs:418-597) ----------------------------------
// From the trees' dense grids ([tree][y][z][x], side 2^d <= 64): voxel counts per value, the sorted
// list of present values, then the bits of every non-default voxel in the 64^3 builder's three
// planes (YZ [y][z] -> x bits, XZ [z][x] -> y bits, XY [y][x] -> z bits), globally and per material.
// OR-ing voxel bits equals fill_masks_for_region's region fills (each region is a cube of voxels).
constexpr uint32_t kOccAll = 3 * 64 * 64;

template <class T>
__global__ void __launch_bounds__(kThreads) occupancy_hist_kernel(const T *grids, uint64_t n_vox,
                                                                   unsigned long long *counts) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const unsigned lane = threadIdx.x & 31u;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n_vox; base += stride) {
        const uint64_t i = base + threadIdx.x;
        const uint32_t v = i < n_vox ? (uint32_t)grids[i] : 0u;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, v);
        if (v != 0 && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(counts + v, (unsigned long long)__popc(peers));
    }
}

// One CTA: slot[v] = rank of v among the present values (ascending), or ~0u.
__global__ void __launch_bounds__(1024) occupancy_index_kernel(const unsigned long long *counts, uint32_t n_values,
                                                               uint32_t *slot, uint32_t *ids,
                                                               unsigned long long *mcounts, uint32_t *n_out) {
    __shared__ uint32_t part[1024];
    const uint32_t per = (n_values + blockDim.x - 1) / blockDim.x;
    const uint32_t v0 = threadIdx.x * per;
    uint32_t c = 0;
    for (uint32_t v = v0; v < v0 + per && v < n_values; ++v) c += (v != 0 && counts[v] != 0) ? 1u : 0u;
    part[threadIdx.x] = c;
    __syncthreads();
    for (uint32_t off = 1; off < blockDim.x; off <<= 1) {  // inclusive scan (Hillis-Steele)
        const uint32_t y = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += y;
        __syncthreads();
    }
    uint32_t r = part[threadIdx.x] - c;
    for (uint32_t v = v0; v < v0 + per && v < n_values; ++v) {
        if (v != 0 && counts[v] != 0) {
            slot[v] = r;
            ids[r] = v;
            mcounts[r] = counts[v];
            ++r;
        } else {
            slot[v] = ~0u;
        }
    }
    if (threadIdx.x == blockDim.x - 1) *n_out = part[threadIdx.x];
}

// Column form of the mask kernels: one thread per line of a tree's grid (a row along x, a column
// along y or along z; orientation o = 0, 1, 2 for the YZ, XZ and XY planes), which builds the line's
// occupancy bits in registers and ORs them into the builder's plane word with one atomic; the same for
// each material present on the line (up to kLineMats tracked in registers, else every material of the
// builder in turn).
constexpr int kLineMats = 6;

template <class T>
__global__ void __launch_bounds__(kThreads) occupancy_lines_kernel(DevInterner I, const T *grids, uint32_t n_trees,
                                                                    int d, const uint32_t *offsets,
                                                                    const uint32_t *slot, const uint32_t *n_mat,
                                                                    uint32_t mat_cap,
                                                                    unsigned long long *global,
                                                                    unsigned long long *per_mat) {
    const uint32_t S = 1u << d;
    const uint64_t lines_per_tree = 3ull * S * S;
    const uint64_t n_lines = lines_per_tree * n_trees;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    bool bad = false;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_lines; i += stride) {
        const uint32_t t = (uint32_t)(i / lines_per_tree), w = (uint32_t)(i % lines_per_tree);
        const uint32_t o = w / (S * S), ab = w % (S * S), a = ab / S, bb = ab % S;
        const uint32_t ox = offsets[3 * t], oy = offsets[3 * t + 1], oz = offsets[3 * t + 2];
        if (ox + S > 64 || oy + S > 64 || oz + S > 64) {
            bad = true;
            continue;
        }
        const T *g = grids + (uint64_t)t * S * S * S;
        // line origin and step in the [y][z][x] grid, target word and the line's bit offset
        uint64_t base, step;
        uint32_t word, shift;
        if (o == 0) {  // YZ[y][z] <- x bits: a = y, bb = z
            base = ((uint64_t)a * S + bb) * S;
            step = 1;
            word = 0 * 4096 + (oy + a) * 64 + (oz + bb);
            shift = ox;
        } else if (o == 1) {  // XZ[z][x] <- y bits: a = z, bb = x
            base = (uint64_t)a * S + bb;
            step = (uint64_t)S * S;
            word = 1 * 4096 + (oz + a) * 64 + (ox + bb);
            shift = oy;
        } else {  // XY[y][x] <- z bits: a = y, bb = x
            base = (uint64_t)a * S * S + bb;
            step = S;
            word = 2 * 4096 + (oy + a) * 64 + (ox + bb);
            shift = oz;
        }
        uint64_t occ = 0;
        uint32_t mv[kLineMats];
        uint64_t mm[kLineMats];
        int nm = 0;
        bool overflow = false;
        for (uint32_t k = 0; k < S; ++k) {
            const uint32_t v = g[base + k * step];
            if (!v) continue;
            occ |= 1ull << k;
            int j = 0;
            while (j < nm && mv[j] != v) ++j;
            if (j == nm) {
                if (nm < kLineMats) {
                    mv[nm] = v;
                    mm[nm] = 0;
                    ++nm;
                } else {
                    overflow = true;
                    continue;
                }
            }
            mm[j] |= 1ull << k;
        }
        if (!occ) continue;
        atomicOr(global + word, (unsigned long long)(occ << shift));
        if (!overflow) {
            for (int j = 0; j < nm; ++j) {
                const uint32_t m = slot[mv[j]];
                if (m < mat_cap) atomicOr(per_mat + (size_t)m * kOccAll + word, (unsigned long long)(mm[j] << shift));
            }
        } else {  // more materials on this line than tracked: one pass per material of the builder
            const uint32_t nmb = *n_mat < mat_cap ? *n_mat : mat_cap;
            for (uint32_t m = 0; m < nmb; ++m) {
                uint64_t bits = 0;
                for (uint32_t k = 0; k < S; ++k) {
                    const uint32_t v = g[base + k * step];
                    if (v && slot[v] == m) bits |= 1ull << k;
                }
                if (bits) atomicOr(per_mat + (size_t)m * kOccAll + word, (unsigned long long)(bits << shift));
            }
        }
    }
    if (bad) set_error(I, ERR_OOB, 54);
}

// active[0..5] (mesh.rs:453-463): the occupied y, z, z, x, y, x coordinates.
__global__ void __launch_bounds__(kThreads) occupancy_active_kernel(const unsigned long long *global,
                                                                    unsigned long long *active) {
    __shared__ unsigned long long acc[3];
    if (threadIdx.x < 3) acc[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long xs = 0, ys = 0, zs = 0;
    for (uint32_t k = threadIdx.x; k < 4096; k += blockDim.x) {
        xs |= global[k];         // YZ words hold x bits
        ys |= global[4096 + k];  // XZ words hold y bits
        zs |= global[8192 + k];  // XY words hold z bits
    }
    atomicOr(&acc[0], xs);
    atomicOr(&acc[1], ys);
    atomicOr(&acc[2], zs);
    __syncthreads();
    if (threadIdx.x == 0) {
        active[0] = acc[1];  // YZ rows: y
        active[1] = acc[2];  // YZ cols: z
        active[2] = acc[2];  // XZ rows: z
        active[3] = acc[0];  // XZ cols: x
        active[4] = acc[1];  // XY rows: y
        active[5] = acc[0];  // XY cols: x
    }
}

// ---- batched occupancy masks, 8-bit voxels: one CTA per builder ---------------------------------------
//
// The output is the work: 98 KB of plane words for each builder and the same again for each material
// slot, so every word is written once, whole and coalesced, and zero slots are not cleared first. A CTA
// keeps the YZ planes ([y][z] -> x bits) of up to three materials in shared memory, filled from the rows of
// its trees' dense grids (a byte compare of 4 voxels at a time gives 4 mask bits); the other two planes
// are bit transposes of it: XY ([y][x] -> z bits) of the 64 x 64 matrix of one y, XZ ([z][x] -> y bits) of
// one z, each by one warp with 5 shuffle steps. The global planes are the OR of the materials' (up to
// three materials) or a plane of their own. Rows of 65 words keep the transposes' column reads free of
// bank conflicts; 100 KB leave two CTAs to an SM, one writing while the other reads.
// 4096 dune chunks in 1024 builders, 8 material slots (906 MB): 302 us with the dense expansion, 1750 us
// when separate kernels counted voxels (one atomic a warp and value, 812 us), cleared the outputs
// (137 us) and ORed every line's bits into them with atomics (607 us).
// Calls with fewer builders than SMs take 1024 threads for each: what bounds them is one CTA's share of the rows
// (13 builders of 16 trees of depth 4 51.8 us against 55.4).
constexpr int kOccManyThreads = 512, kOccFewThreads = 1024;
constexpr int kOccPlanes = 3;                 // YZ planes held at once
constexpr uint32_t kOccPitch = 65;            // words of a plane's row in shared memory
constexpr uint32_t kOccPlaneWords = 64 * kOccPitch;
constexpr size_t kOccSmem = kOccPlanes * kOccPlaneWords * 8;
constexpr uint32_t kNoTree = 0xFFFFFFFFu;
constexpr uint32_t kOccAny = 0u;              // plane of the non-default voxels (0 is no material)
constexpr uint32_t kOccNone = 0xFFFFFFFFu;    // unused plane

// Lists the trees of each builder, in any order: the first kOccListed of them side by side in listed, with their
// number less one in head[n_builders + builder], the others linked, head[builder] -> next[tree] -> ...
constexpr uint32_t kOccListed = 64;
__global__ void __launch_bounds__(kThreads) occupancy_link_kernel(DevInterner I, uint32_t n_trees,
                                                                   const uint32_t *builder_of, uint32_t n_builders,
                                                                   uint32_t *head, uint32_t *next, uint32_t *listed) {
    bool bad = false;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n_trees; t += gridDim.x * blockDim.x) {
        const uint32_t b = builder_of[t];
        if (b >= n_builders) {
            bad = true;
            continue;
        }
        const uint32_t k = atomicAdd(head + n_builders + b, 1u) + 1u;
        if (k < kOccListed)
            listed[(size_t)b * kOccListed + k] = t;
        else
            next[t] = atomicExch(head + b, t);
    }
    if (bad) set_error(I, ERR_OOB, 54);
}

// In place: lane r holds row r of a 32 x 32 bit matrix before and after its transpose. Whole warp.
__device__ __forceinline__ uint32_t transpose32(uint32_t v) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t m = 0x0000FFFFu;  // the columns without bit s
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, v, s);
        v = (lane & s) ? (v & ~m) | ((y >> s) & m) : (v & m) | ((y & m) << s);
        m ^= m << (s >> 1);
    }
    return v;
}

// Transpose of a 64 x 64 bit matrix: the lane holds rows lane (a) and lane + 32 (b) before and after.
__device__ __forceinline__ void transpose64(uint64_t &a, uint64_t &b) {
    if (!__any_sync(0xFFFFFFFFu, (a | b) != 0)) return;
    const uint32_t a0 = transpose32((uint32_t)a), a1 = transpose32((uint32_t)(a >> 32));
    const uint32_t b0 = transpose32((uint32_t)b), b1 = transpose32((uint32_t)(b >> 32));
    a = a0 | ((uint64_t)b0 << 32);
    b = a1 | ((uint64_t)b1 << 32);
}

// Bit k of the result: byte k of w equals byte k of splat.
__device__ __forceinline__ uint32_t equal_bytes(uint32_t w, uint32_t splat) {
    const uint32_t x = w ^ splat;
    const uint32_t z = ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu) >> 7;  // 1 in each equal byte
    return (z * 0x01020408u) >> 24;
}

// Calls f(k, w, n) for the words of 16 voxels v, the 4q-th word of their row on: w is the 4 voxels from 4k on, and
// holds for n voxels (16 when it repeats, one value along x being the usual case, else 4).
template <class F>
__device__ __forceinline__ void quad_words(uint32_t q, uint4 v, F f) {
    if (v.x == v.y && v.x == v.z && v.x == v.w) {
        f(4 * q, v.x, 16u);
    } else {
        f(4 * q, v.x, 4u);
        f(4 * q + 1, v.y, 4u);
        f(4 * q + 2, v.z, 4u);
        f(4 * q + 3, v.w, 4u);
    }
}

// The same for a row of S voxels in order. A row of 2 voxels is padded with zeros.
template <class F>
__device__ __forceinline__ void row_words(const uint8_t *row, uint32_t S, F f) {
    if (S >= 16) {
        for (uint32_t q = 0; q < S / 16; ++q) quad_words(q, __ldg(reinterpret_cast<const uint4 *>(row) + q), f);
    } else if (S >= 4) {
        for (uint32_t k = 0; k < S / 4; ++k) f(k, __ldg(reinterpret_cast<const uint32_t *>(row) + k), 4u);
    } else {
        f(0, (uint32_t)__ldg(reinterpret_cast<const uint16_t *>(row)), 4u);
    }
}

// Calls begin(), then f for a row's words, then end(q) for the thread's rows q of [0, n). Rows of 16 voxels are one
// load each: four of them are under way at a time.
template <class Row, class Begin, class F, class End>
__device__ __forceinline__ void each_row(uint32_t n, uint32_t S, Row row_of, Begin begin, F f, End end) {
    if (S == 16) {
        for (uint32_t q0 = threadIdx.x; q0 < n; q0 += 4 * blockDim.x) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t q = q0 + u * blockDim.x;
                if (q < n) v[u] = __ldg(reinterpret_cast<const uint4 *>(row_of(q)));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t q = q0 + u * blockDim.x;
                if (q >= n) break;
                begin();
                quad_words(0, v[u], f);
                end(q);
            }
        }
        return;
    }
    for (uint32_t q = threadIdx.x; q < n; q += blockDim.x) {
        begin();
        row_words(row_of(q), S, f);
        end(q);
    }
}

// Two words at p (p[0], p[1]); wide: p is 16-byte aligned. The outputs are stored evict-first: they are several
// times the L2's size, and the grids that the next sweep reads should stay there.
__device__ __forceinline__ void store_words(unsigned long long *p, ulonglong2 v, bool wide) {
    if (wide) {
        __stcs(reinterpret_cast<ulonglong2 *>(p), v);
    } else {
        __stcs(p, v.x);
        __stcs(p + 1, v.y);
    }
}

template <int kOccThreads>
__global__ void __launch_bounds__(kOccThreads, 1024 / kOccThreads) occupancy_builders_kernel(
    DevInterner I, const uint8_t *grids, int d, const uint32_t *offsets, const uint32_t *head, const uint32_t *next,
    const uint32_t *listed, uint32_t max_mat, uint32_t *ids, unsigned long long *mcounts, uint32_t *n_mat_out, unsigned long long *global,
    unsigned long long *per_mat, unsigned long long *active) {
    extern __shared__ __align__(16) unsigned long long occ_planes[];
    __shared__ uint8_t present[256];
    __shared__ uint32_t mat[256];  // present materials, ascending
    __shared__ uint32_t n_mat_s, cnt_s[kOccPlanes], act_s[6];
    __shared__ uint32_t list_s[kOccListed], ofs_s[kOccListed], list_n, list_next;  // some trees of the builder
    const uint32_t b = blockIdx.x;
    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t S = 1u << d, rows = S * S;
    const uint64_t per_tree = 1ull << (3 * d);
    // Up to kOccListed trees and their offsets (x, y, z a byte each; all ones: outside) to shared memory: the first
    // ones together, the linked ones by one thread. A sweep takes the rows of all of them side by side: 16 trees of
    // depth 4 walked one after the other, by 256 of the 512 threads, took 70.0 us against 55.4.
    const auto offsets_of = [&](uint32_t t) {
        const uint32_t x = offsets[3 * t], y = offsets[3 * t + 1], z = offsets[3 * t + 2];
        return x <= 64 - S && y <= 64 - S && z <= 64 - S ? x | y << 8 | z << 16 : 0xFFFFFFFFu;
    };
    bool whole = false;  // all of them are there
    const auto load_trees = [&](bool first) {
        if (whole) return list_n;
        __syncthreads();
        if (first) {
            const uint32_t t = tid < kOccListed ? listed[(size_t)b * kOccListed + tid] : 0u;  // beside their number
            const uint32_t n = min(head[gridDim.x + b] + 1u, kOccListed);
            if (tid < n) {
                list_s[tid] = t;
                ofs_s[tid] = offsets_of(t);
            }
            if (tid == 0) {
                list_n = n;
                list_next = head[b];
            }
        } else if (tid == 0) {
            uint32_t n = 0, t = list_next;
            for (; t != kNoTree && n < kOccListed; t = next[t], ++n) {
                list_s[n] = t;
                ofs_s[n] = offsets_of(t);
            }
            list_n = n;
            list_next = t;
        }
        __syncthreads();
        whole = first && list_next == kNoTree;
        return list_n;
    };
    const bool wide = ((reinterpret_cast<uintptr_t>(global) | reinterpret_cast<uintptr_t>(per_mat)) & 15u) == 0;
    unsigned long long *gout = global + (size_t)b * kOccAll, *mout = per_mat + (size_t)b * max_mat * kOccAll;
    if (tid < 256) present[tid] = 0;
    if (tid < 6) act_s[tid] = 0;
    __syncthreads();
    // the values present: idempotent byte stores, most words repeat the thread's last value
    uint32_t last = 0;
    const auto row_of = [&](uint32_t q) { return grids + list_s[q >> (2 * d)] * per_tree + (size_t)(q & (rows - 1)) * S; };
    for (uint32_t n = load_trees(true); n; n = list_next != kNoTree ? load_trees(false) : 0u)
        each_row(n * rows, S, row_of, [] {}, [&](uint32_t, uint32_t w, uint32_t) {
            if (w == last) return;
#pragma unroll
            for (int k = 0; k < 4; ++k) present[(w >> (8 * k)) & 0xFFu] = 1;
            last = w;
        }, [](uint32_t) {});
    __syncthreads();
    if (warp == 0) {
        uint32_t n = 0;
        for (uint32_t v0 = 0; v0 < 256; v0 += 32) {
            const uint32_t v = v0 + lane;
            const bool p = v != 0 && present[v];
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, p);
            const uint32_t k = n + __popc(bal & ((1u << lane) - 1u));
            if (p) {
                mat[k] = v;
                if (k < max_mat) ids[(size_t)b * max_mat + k] = v;
            }
            n += __popc(bal);
        }
        if (lane == 0) {
            n_mat_s = n;
            n_mat_out[b] = n;
        }
    }
    __syncthreads();
    const uint32_t n_mat = n_mat_s, stored = n_mat < max_mat ? n_mat : max_mat;
    for (uint32_t k = stored; k < max_mat; ++k) {  // slots without a material
        unsigned long long *z = mout + (size_t)k * kOccAll;
        for (uint32_t i = 2 * tid; i < kOccAll; i += 2 * kOccThreads) store_words(z + i, make_ulonglong2(0, 0), wide);
    }
    const bool by_or = n_mat <= kOccPlanes;  // the global planes are the OR of the materials'
    bool bad = false;
    uint64_t ax = 0, ay = 0, az = 0;  // occupied coordinates seen by this thread
    // sweeps over the trees, kOccPlanes planes each: with by_or the materials, else [any, material 0, ...]
    const uint32_t n_planes = by_or ? n_mat : stored + 1;
    for (uint32_t p0 = 0; p0 == 0 || p0 < n_planes; p0 += kOccPlanes) {
        uint32_t want[kOccPlanes], splat[kOccPlanes], acc[kOccPlanes];
        unsigned long long *out[kOccPlanes];  // where a plane goes, null: nowhere
#pragma unroll
        for (int p = 0; p < kOccPlanes; ++p) {
            const uint32_t i = p0 + p;
            want[p] = kOccNone;
            out[p] = nullptr;
            acc[p] = 0;
            if (i < n_planes) {
                const uint32_t k = by_or ? i : i - 1;  // material index
                want[p] = (!by_or && i == 0) ? kOccAny : mat[k];
                if (want[p] == kOccAny)
                    out[p] = gout;
                else if (k < stored)
                    out[p] = mout + (size_t)k * kOccAll;
            }
            splat[p] = want[p] * 0x01010101u;
        }
        if (tid < kOccPlanes) cnt_s[tid] = 0;
        for (uint32_t i = tid; i < kOccPlanes * kOccPlaneWords; i += kOccThreads) occ_planes[i] = 0;
        __syncthreads();
        uint64_t m[kOccPlanes];
        for (uint32_t n = load_trees(true); n; n = list_next != kNoTree ? load_trees(false) : 0u)
            each_row(n * rows, S, row_of, [&] {
#pragma unroll
                for (int p = 0; p < kOccPlanes; ++p) m[p] = 0;
            }, [&](uint32_t k, uint32_t w, uint32_t n_same) {
                if (w == 0) return;
#pragma unroll
                for (int p = 0; p < kOccPlanes; ++p) {
                    if (want[p] == kOccNone) continue;
                    uint32_t e = equal_bytes(w, splat[p]);
                    if (want[p] == kOccAny) e ^= 0xFu;
                    if (n_same == 16) e *= 0x1111u;
                    m[p] |= (uint64_t)e << (4 * k);
                }
            }, [&](uint32_t q) {
                const uint32_t at_tree = ofs_s[q >> (2 * d)], r = q & (rows - 1);
                const bool inside = at_tree != 0xFFFFFFFFu;
                const uint32_t ox = at_tree & 0xFFu, oy = at_tree >> 8 & 0xFFu, oz = at_tree >> 16;
                bad = bad || !inside;
                uint32_t *at = reinterpret_cast<uint32_t *>(occ_planes) +
                               (inside ? 2 * ((oy + (r >> d)) * kOccPitch + oz + (r & (S - 1))) : 0u);
#pragma unroll
                for (int p = 0; p < kOccPlanes; ++p) {
                    acc[p] += __popcll(m[p]);
                    const uint64_t bits = inside ? m[p] << ox : 0ull;
                    if (bits) {
                        uint32_t *w = at + 2 * p * kOccPlaneWords;
                        if ((uint32_t)bits) atomicOr(w, (uint32_t)bits);
                        if (bits >> 32) atomicOr(w + 1, (uint32_t)(bits >> 32));
                    }
                }
            });
#pragma unroll
        for (int p = 0; p < kOccPlanes; ++p) {
            const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, acc[p]);
            if (lane == 0 && n) atomicAdd(cnt_s + p, n);
        }
        __syncthreads();
        if (tid < kOccPlanes) {  // tid is the plane
            const uint32_t i = p0 + tid;
            const uint32_t k = by_or ? i : i - 1;
            if (i < n_planes && (by_or || i > 0) && k < stored) mcounts[(size_t)b * max_mat + k] = cnt_s[tid];
        }
        const bool with_global = p0 == 0;
        // YZ planes: two words a thread
        for (uint32_t i = 2 * tid; i < 4096; i += 2 * kOccThreads) {
            const uint32_t at = (i >> 6) * kOccPitch + (i & 63u);
            ulonglong2 any = make_ulonglong2(0, 0);
#pragma unroll
            for (int p = 0; p < kOccPlanes; ++p) {
                const ulonglong2 v = make_ulonglong2(occ_planes[p * kOccPlaneWords + at], occ_planes[p * kOccPlaneWords + at + 1]);
                any.x |= v.x;
                any.y |= v.y;
                if (out[p]) store_words(out[p] + i, v, wide);
            }
            if (with_global) {
                if (by_or) store_words(gout + i, any, wide);
                ax |= any.x | any.y;
            }
        }
        // XY planes from the matrix of one y, XZ planes from that of one z, a warp each
        for (uint32_t f = warp; f < 128; f += kOccThreads / 32) {
            const bool xz = f >= 64;
            const uint32_t k = f & 63u;
            const uint32_t at = xz ? lane * kOccPitch + k : k * kOccPitch + lane;
            const uint32_t step = xz ? 32 * kOccPitch : 32;
            const uint32_t word = (xz ? 4096 : 8192) + 64 * k + lane;
            uint64_t ga = 0, gb = 0;
#pragma unroll
            for (int p = 0; p < kOccPlanes; ++p) {
                uint64_t u = occ_planes[p * kOccPlaneWords + at], v = occ_planes[p * kOccPlaneWords + at + step];
                if (want[p] == kOccNone) continue;
                transpose64(u, v);
                ga |= u;
                gb |= v;
                if (out[p]) {
                    __stcs(out[p] + word, (unsigned long long)u);
                    __stcs(out[p] + word + 32, (unsigned long long)v);
                }
            }
            if (with_global) {
                if (by_or) {
                    __stcs(gout + word, (unsigned long long)ga);
                    __stcs(gout + word + 32, (unsigned long long)gb);
                }
                if (xz)
                    ay |= ga | gb;
                else
                    az |= ga | gb;
            }
        }
        __syncthreads();  // the planes are cleared by the next sweep
    }
    const uint64_t ac[3] = {ax, ay, az};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const uint32_t w = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(ac[k >> 1] >> (32 * (k & 1))));
        if (lane == 0 && w) atomicOr(act_s + k, w);
    }
    __syncthreads();
    if (tid < 6) {  // the occupied y, z, z, x, y, x coordinates (mesh.rs:453-463)
        const int src[6] = {1, 2, 2, 0, 1, 0};
        const int k = src[tid];
        active[6 * (size_t)b + tid] = act_s[2 * k] | ((unsigned long long)act_s[2 * k + 1] << 32);
    }
    if (bad) set_error(I, ERR_OOB, 54);
}

// ---- model serialisation (VoxModel::serialize, world/voxmodel.rs:177-282; serialize_chunk,
// world/voxchunk.rs:382-405) ------------------------------------------------------------------------
// Live leaves and live branches other than EMPTY are renumbered in slot-index order (leaves 1..L,
// then branches L+1..), each record's byte length is computed in parallel, exclusive scans place
// the records, and every node writes its own record: varint(new id) then the value (leaves), or
// varint(new id), mask, varint(new id) of each non-empty child and the LOD value (branches); values
// big-endian. Chunk records: "VoxTreeChunk", position (3 x i32 BE), varint(new id of the root).
__device__ __forceinline__ uint32_t varint_len(uint32_t v) {
    uint32_t n = 1;
    while (v >= 0x80u) {
        v >>= 7;
        ++n;
    }
    return n;
}

__device__ __forceinline__ uint8_t *put_varint(uint8_t *p, uint32_t v) {
    while (v >= 0x80u) {
        *p++ = (uint8_t)((v & 0x7Fu) | 0x80u);
        v >>= 7;
    }
    *p++ = (uint8_t)v;
    return p;
}

__device__ __forceinline__ uint8_t *put_value_be(uint8_t *p, uint32_t v, int vb) {
    if (vb == 2) *p++ = (uint8_t)(v >> 8);
    *p++ = (uint8_t)v;
    return p;
}

// Plan of one serialisation, in device scratch. Two scans (ranks, then record offsets) of (leaf, branch)
// pairs over the slots [1, next_index): a CTA owns a contiguous range, one launch sums the ranges, the next
// starts each range from the sum of the ranges before it. Work follows the slots handed out, not the
// capacity, and no CTA waits for another. (Classifying, numbering and scanning every slot of the budget
// took 16 launches and 300 us at 3.4 M slots, and one thread summed and wrote the chunk records: 840 us
// for 1024 chunks.)
struct SerBufs {
    uint32_t *rank, *off;           // per slot: rank among the leaves or branches; offset of its record in its table
    ulonglong2 *part;               // [scan][range] sums
    unsigned long long *total;      // leaves, branches, bytes of the leaf table, bytes of the branch table
    unsigned long long *chunk_off;  // per chunk: offset of its record in the chunk section
    size_t words;                   // u32 words of the whole scratch
    SerBufs(const DevInterner &I, uint32_t n_chunks, void *w);
};
constexpr uint32_t kSerRanges = 608;  // most ranges (CTAs) of a scan: four to an SM

// The slots of range blockIdx.x: whole CTA widths, so a small model spreads over many CTAs.
__device__ __forceinline__ void ser_range(uint32_t n, uint32_t &lo, uint32_t &hi) {
    const uint64_t per = ((((uint64_t)n + gridDim.x - 1) / gridDim.x + kThreads - 1) / kThreads) * kThreads;
    const uint64_t l = blockIdx.x * per;
    lo = l < n ? (uint32_t)l : n;
    hi = l + per < n ? (uint32_t)(l + per) : n;
}

// Sum over the CTA of (leaf, branch) pairs, in every thread. Every thread of the CTA calls it.
__device__ __forceinline__ ulonglong2 ser_cta_sum(ulonglong2 v) {
    __shared__ ulonglong2 warp_sum[kThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xFFFFFFFFu, v.x, o);
        v.y += __shfl_xor_sync(0xFFFFFFFFu, v.y, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) warp_sum[threadIdx.x >> 5] = v;
    __syncthreads();
    ulonglong2 all = make_ulonglong2(0, 0);
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        all.x += warp_sum[w].x;
        all.y += warp_sum[w].y;
    }
    return all;
}

// The new id of a node: leaves 1..L in slot order, then the branches; EMPTY is 0.
__device__ __forceinline__ uint32_t ser_new_id(const DevInterner &I, const SerBufs &b, uint64_t id) {
    if (id == EMPTY_ID) return 0;
    return b.rank[id_index(id)] + 1u + (id_is_leaf(id) ? 0u : (uint32_t)b.total[0]);
}

// Sums of the ranges. scan 0: live nodes; scan 1: lengths of their records (left in off[]).
__global__ void __launch_bounds__(kThreads) ser_sum_kernel(DevInterner I, SerBufs b, int scan) {
    const uint32_t n = (uint32_t)I.ctr->next_index, vb = I.vbits / 8;  // slot 0 is EMPTY
    uint32_t lo, hi;
    ser_range(n, lo, hi);
    ulonglong2 sum = make_ulonglong2(0, 0);
    for (uint64_t i = (uint64_t)lo + threadIdx.x; i < hi; i += kThreads) {
        const uint64_t id = i ? I.ids[i] : 0ull;
        if (id == 0) continue;
        uint32_t v = 1;
        if (scan == 1) {
            v = varint_len(ser_new_id(I, b, id)) + vb;
            if (!id_is_leaf(id)) {
                v += 1;
                const ulonglong2 *c = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * i);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ulonglong2 w = c[j];
                    if (w.x != EMPTY_ID) v += varint_len(ser_new_id(I, b, w.x));
                    if (w.y != EMPTY_ID) v += varint_len(ser_new_id(I, b, w.y));
                }
            }
            b.off[i] = v;
        }
        if (id_is_leaf(id))
            sum.x += v;
        else
            sum.y += v;
    }
    sum = ser_cta_sum(sum);
    if (threadIdx.x == 0) b.part[scan * kSerRanges + blockIdx.x] = sum;
}

// Exclusive prefixes of the scan into rank[] (0) or off[] (1), and the totals.
__global__ void __launch_bounds__(kThreads) ser_prefix_kernel(DevInterner I, SerBufs b, int scan) {
    __shared__ uint2 warp_sum[kThreads / 32];
    const uint32_t n = (uint32_t)I.ctr->next_index;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const ulonglong2 *part = b.part + scan * kSerRanges;
    ulonglong2 run = make_ulonglong2(0, 0);
    for (uint32_t k = threadIdx.x; k < blockIdx.x; k += kThreads) {
        run.x += part[k].x;
        run.y += part[k].y;
    }
    run = ser_cta_sum(run);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        b.total[2 * scan] = run.x + part[blockIdx.x].x;
        b.total[2 * scan + 1] = run.y + part[blockIdx.x].y;
    }
    uint32_t lo, hi;
    ser_range(n, lo, hi);
    uint32_t *out = scan ? b.off : b.rank;
    for (uint64_t base = lo; base < hi; base += kThreads) {  // the same number of rounds in every thread
        const uint64_t i = base + threadIdx.x;
        const uint64_t id = (i > 0 && i < hi) ? I.ids[i] : 0ull;
        const bool leaf = id != 0 && id_is_leaf(id);
        const uint32_t v = id == 0 ? 0u : (scan ? out[i] : 1u);
        uint2 incl = make_uint2(leaf ? v : 0u, leaf ? 0u : v);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl.x, o), y = __shfl_up_sync(0xFFFFFFFFu, incl.y, o);
            if (lane >= (unsigned)o) incl = make_uint2(incl.x + x, incl.y + y);
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        uint2 before = make_uint2(0, 0), all = make_uint2(0, 0);
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) {
            const uint2 x = warp_sum[w];
            if (w < (int)warp) before = make_uint2(before.x + x.x, before.y + x.y);
            all = make_uint2(all.x + x.x, all.y + x.y);
        }
        if (id != 0) out[i] = leaf ? (uint32_t)run.x + before.x + incl.x - v : (uint32_t)run.y + before.y + incl.y - v;
        run.x += all.x;
        run.y += all.y;
        __syncthreads();  // warp_sum is reused by the next round
    }
}

// One CTA: the chunk records' offsets in their section, and the size of the whole payload.
__global__ void __launch_bounds__(1024) ser_chunks_kernel(DevInterner I, SerBufs b, uint32_t n_chunks,
                                                          const uint32_t *trees, unsigned long long *total) {
    __shared__ uint32_t warp_sum[32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long before = 0;
    for (uint32_t base = 0; base < n_chunks; base += 1024) {
        const uint32_t k = base + threadIdx.x;
        uint32_t len = 0;
        if (k < n_chunks) {
            const uint32_t t = trees[k];
            len = 24 + varint_len(ser_new_id(I, b, t < I.tree_cap ? I.roots[t] : EMPTY_ID));
        }
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (unsigned)o) incl += u;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        uint32_t w = warp_sum[lane], wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= (unsigned)o) wi += u;
        }
        const uint32_t mine = __shfl_sync(0xFFFFFFFFu, wi - w, warp), all = __shfl_sync(0xFFFFFFFFu, wi, 31);
        if (k < n_chunks) b.chunk_off[k] = before + mine + incl - len;
        before += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = 12ull + b.total[2] + b.total[3] + before;
}

__device__ __forceinline__ void put_u32_be(uint8_t *p, uint32_t v) {
    p[0] = (uint8_t)(v >> 24);
    p[1] = (uint8_t)(v >> 16);
    p[2] = (uint8_t)(v >> 8);
    p[3] = (uint8_t)v;
}

// The records: out = [u32 L][leaf records][u32 B][branch records][u32 n_chunks][chunk records], a thread
// a node, then a thread a chunk. branch_patterns without EMPTY are counted (the reference writes its
// size - 1).
__global__ void __launch_bounds__(kThreads) ser_write_kernel(DevInterner I, SerBufs b, uint32_t n_chunks,
                                                             const uint32_t *trees, const int32_t *pos, uint8_t *out) {
    const int vb = I.vbits / 8;
    const uint32_t n = (uint32_t)I.ctr->next_index;
    const uint64_t leaf_base = 4, branch_base = 8 + b.total[2], chunk_base = 12 + b.total[2] + b.total[3];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (first == 0) {
        put_u32_be(out, (uint32_t)b.total[0]);
        put_u32_be(out + branch_base - 4, (uint32_t)b.total[1]);
        put_u32_be(out + chunk_base - 4, n_chunks);
    }
    for (uint64_t i = first + 1; i < n; i += stride) {
        const uint64_t id = I.ids[i];
        if (id == 0) continue;
        uint8_t *p = out + (id_is_leaf(id) ? leaf_base : branch_base) + b.off[i];
        p = put_varint(p, ser_new_id(I, b, id));
        if (!id_is_leaf(id)) {
            *p++ = (uint8_t)id_mask(id);
            const uint64_t *c = I.children + 8ull * i;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (c[k] != EMPTY_ID) p = put_varint(p, ser_new_id(I, b, c[k]));
        }
        put_value_be(p, node_value(I, (uint32_t)i), vb);
    }
    const char magic[12] = {'V', 'o', 'x', 'T', 'r', 'e', 'e', 'C', 'h', 'u', 'n', 'k'};
    for (uint64_t k = first; k < n_chunks; k += stride) {
        uint8_t *p = out + chunk_base + b.chunk_off[k];
#pragma unroll
        for (int j = 0; j < 12; ++j) p[j] = (uint8_t)magic[j];
        for (int a = 0; a < 3; ++a) put_u32_be(p + 12 + 4 * a, (uint32_t)pos[3 * k + a]);
        const uint32_t t = trees[k];
        put_varint(p + 24, ser_new_id(I, b, t < I.tree_cap ? I.roots[t] : EMPTY_ID));
    }
}

SerBufs::SerBufs(const DevInterner &I, uint32_t n_chunks, void *w) {
    char *base = static_cast<char *>(w);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char *r = base + at;
        at += (bytes + 15) & ~(size_t)15;
        return r;
    };
    rank = reinterpret_cast<uint32_t *>(take((size_t)I.capacity * 4));
    off = reinterpret_cast<uint32_t *>(take((size_t)I.capacity * 4));
    chunk_off = reinterpret_cast<unsigned long long *>(take((size_t)n_chunks * 8));
    total = reinterpret_cast<unsigned long long *>(take(32));
    part = reinterpret_cast<ulonglong2 *>(take(2 * kSerRanges * sizeof(ulonglong2)));
    words = at / 4;
}

cudaError_t launch_to_dense(const DevInterner &I, const uint32_t *trees, int d, uint64_t cube_begin,
                            uint64_t n_cubes, void *out, int num_sms, cudaStream_t s) {
    if (n_cubes == 0) return cudaSuccess;
    const uint64_t threads = d == 1 ? n_cubes : n_cubes << (3 * (d < 5 ? d - 2 : 3));
    uint64_t blocks = (threads + kDenseOutThreads - 1) / kDenseOutThreads;
    const uint64_t cap = (uint64_t)num_sms * 64;
    if (blocks > cap) blocks = cap;
    count_launches(1);
    auto launch = [&](auto *o) {
        using T = std::remove_pointer_t<decltype(o)>;
        if (d == 1)
            to_dense_depth1_kernel<T><<<(unsigned)blocks, kDenseOutThreads, 0, s>>>(I, trees, cube_begin, n_cubes, o);
        else
            to_dense_kernel<T><<<(unsigned)blocks, kDenseOutThreads, 0, s>>>(I, trees, d, cube_begin, n_cubes, o);
    };
    if (I.vbits == 8)
        launch((uint8_t *)out);
    else
        launch((uint16_t *)out);
    return cudaGetLastError();
}

cudaError_t launch_occupancy(const DevInterner &I, const void *grids, uint32_t n_trees, int d, const uint32_t *offsets,
                             unsigned long long *counts, uint32_t *slot, uint32_t *ids, unsigned long long *mcounts,
                             uint32_t *n_mat, uint32_t mat_cap, unsigned long long *global, unsigned long long *per_mat,
                             unsigned long long *active, int num_sms, cudaStream_t s) {
    const uint64_t n_vox = ((uint64_t)n_trees) << (3 * d);
    uint64_t blocks = (n_vox + kThreads - 1) / kThreads;
    if (blocks > (uint64_t)num_sms * 16) blocks = (uint64_t)num_sms * 16;
    const uint32_t n_values = 1u << I.vbits;
    count_launches(4);
    if (I.vbits == 8)
        occupancy_hist_kernel<uint8_t><<<(unsigned)blocks, kThreads, 0, s>>>((const uint8_t *)grids, n_vox, counts);
    else
        occupancy_hist_kernel<uint16_t><<<(unsigned)blocks, kThreads, 0, s>>>((const uint16_t *)grids, n_vox, counts);
    occupancy_index_kernel<<<1, 1024, 0, s>>>(counts, n_values, slot, ids, mcounts, n_mat);
    uint64_t lblocks = ((3ull * n_trees << (2 * d)) + kThreads - 1) / kThreads;
    if (lblocks > (uint64_t)num_sms * 16) lblocks = (uint64_t)num_sms * 16;
    if (I.vbits == 8)
        occupancy_lines_kernel<uint8_t><<<(unsigned)lblocks, kThreads, 0, s>>>(
            I, (const uint8_t *)grids, n_trees, d, offsets, slot, n_mat, mat_cap, global, per_mat);
    else
        occupancy_lines_kernel<uint16_t><<<(unsigned)lblocks, kThreads, 0, s>>>(
            I, (const uint16_t *)grids, n_trees, d, offsets, slot, n_mat, mat_cap, global, per_mat);
    occupancy_active_kernel<<<1, kThreads, 0, s>>>(global, active);
    return cudaGetLastError();
}

size_t occupancy_listed_words(uint32_t n_builders) { return (size_t)n_builders * kOccListed; }

size_t serialize_scratch_words(const DevInterner &I, uint32_t n_chunks) { return SerBufs(I, n_chunks, nullptr).words; }

cudaError_t launch_serialize_plan(const DevInterner &I, uint32_t *w, uint32_t n_chunks, const uint32_t *trees,
                                  unsigned long long *total, int num_sms, cudaStream_t s) {
    const SerBufs b(I, n_chunks, w);
    const unsigned g = std::min<unsigned>((unsigned)num_sms * 4, kSerRanges);
    count_launches(5);
    for (int scan = 0; scan < 2; ++scan) {
        ser_sum_kernel<<<g, kThreads, 0, s>>>(I, b, scan);
        ser_prefix_kernel<<<g, kThreads, 0, s>>>(I, b, scan);
    }
    ser_chunks_kernel<<<1, 1024, 0, s>>>(I, b, n_chunks, trees, total);
    return cudaGetLastError();
}

cudaError_t launch_serialize_write(const DevInterner &I, uint32_t *w, uint32_t n_chunks, const uint32_t *trees,
                                   const int32_t *pos, uint8_t *out, int num_sms, cudaStream_t s) {
    const SerBufs b(I, n_chunks, w);
    count_launches(1);
    ser_write_kernel<<<(unsigned)num_sms * 8, kThreads, 0, s>>>(I, b, n_chunks, trees, pos, out);
    return cudaGetLastError();
}

cudaError_t launch_occupancy_many(const DevInterner &I, const uint8_t *grids, uint32_t n_trees, int d,
                                  const uint32_t *builder_of, const uint32_t *offsets, uint32_t n_builders,
                                  uint32_t *head, uint32_t *next, uint32_t *listed, uint32_t max_mat, uint32_t *ids,
                                  unsigned long long *mcounts, uint32_t *n_mat, unsigned long long *global,
                                  unsigned long long *per_mat, unsigned long long *active, int num_sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(head, 0xFF, (size_t)n_builders * 8, s);
    if (e != cudaSuccess) return e;
    const bool few = n_builders < (uint32_t)num_sms;
    const auto kernel = few ? occupancy_builders_kernel<kOccFewThreads> : occupancy_builders_kernel<kOccManyThreads>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOccSmem);
    if (e != cudaSuccess) return e;
    uint64_t blocks = ((uint64_t)n_trees + kThreads - 1) / kThreads;
    if (blocks > (uint64_t)num_sms * 8) blocks = (uint64_t)num_sms * 8;
    count_launches(2);
    occupancy_link_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(I, n_trees, builder_of, n_builders, head, next,
                                                              listed);
    kernel<<<n_builders, few ? kOccFewThreads : kOccManyThreads, kOccSmem, s>>>(I, grids, d, offsets, head, next, listed, max_mat, ids,
                                                                        mcounts, n_mat, global, per_mat, active);
    return cudaGetLastError();
}

// Levels the table of a call skips (0: no table). n queries over n_trees trees: no more entries than an
// eighth of the queries, so that filling them stays small beside the reads, and than kGetTableEntries; from
// two levels up, since one saves no more than it costs; and not for calls so small that the extra launch
// shows. A call and its wait on a tree of depth 9: 31.4 us with the table and 31.4 without for 524 K gets, 35.1 and
// 37.4 for 1 M, 59 and 76 for 4 M; on 1000 trees of depth 4 30.6 and 28.3, 33.0 and 32.2, 51 and 54.
int get_table_levels(uint64_t n, uint32_t n_trees, int max_depth) {
    if (n < (1u << 20) || n_trees == 0) return 0;
    const uint64_t most = std::min<uint64_t>(kGetTableEntries, n / 8);
    int k = 0;
    while (k < max_depth && ((uint64_t)n_trees << (3 * (k + 1))) <= most) ++k;
    return k >= 2 ? k : 0;
}

cudaError_t launch_get_many(const DevInterner &I, uint64_t n, const uint32_t *trees, const int32_t *xyz,
                            uint8_t *found, void *values, uint64_t *table, int k, uint32_t n_trees, int num_sms,
                            cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    uint64_t blocks = (n + kThreads - 1) / kThreads;
    const uint64_t cap = (uint64_t)num_sms * 64;
    if (blocks > cap) blocks = cap;
    const unsigned g = (unsigned)blocks;
    if (k > 0) {
        uint64_t tb = (((uint64_t)n_trees << (3 * k)) + kThreads - 1) / kThreads;
        if (tb > cap) tb = cap;
        count_launches(1);
        get_table_kernel<<<(unsigned)tb, kThreads, 0, s>>>(I, n_trees, k, table);
    }
    count_launches(1);
    auto launch = [&](auto *v) -> cudaError_t {
        using T = std::remove_pointer_t<decltype(v)>;
        if (k > 0)
            return launch_pdl(get_kernel<T, true>, dim3(g), dim3(kThreads), 0, s, I, n, trees, xyz, found, v,
                              (const uint64_t *)table, k, n_trees);
        get_kernel<T, false><<<g, kThreads, 0, s>>>(I, n, trees, xyz, found, v, nullptr, 0, 0);
        return cudaGetLastError();
    };
    return I.vbits == 8 ? launch((uint8_t *)values) : launch((uint16_t *)values);
}

cudaError_t launch_release(const DevInterner &I, uint64_t *list, uint32_t *frontier_a, uint32_t *frontier_b,
                           int rounds, int num_sms, cudaStream_t s, bool may_wait) {
    DevInterner Ic = I;
    const uint64_t *l = list;
    int wait = may_wait ? 1 : 0;
    void *args[] = {&Ic, &l, &frontier_a, &frontier_b, &rounds, &wait};
    count_launches(1);
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(release_kernel), dim3((unsigned)num_sms * kReleaseCtas),
                                       dim3(kThreads), args, release_smem(I.vbits), s);
}

cudaError_t launch_tree_get(const DevInterner &I, uint32_t tree, int32_t x, int32_t y, int32_t z, HostReply *r, cudaStream_t s) {
    count_launches(1);
    tree_get_kernel<<<1, 1, 0, s>>>(I, tree, x, y, z, r);
    return cudaGetLastError();
}

cudaError_t launch_tree_set(const DevInterner &I, uint32_t tree, int32_t x, int32_t y, int32_t z, uint32_t v,
                            uint64_t *queue, uint64_t queue_cap, HostReply *r, cudaStream_t s) {
    count_launches(1);
    tree_set_kernel<<<1, kSetThreads, 0, s>>>(I, tree, x, y, z, v, queue, queue_cap, r);
    return cudaGetLastError();
}

// Four calls a tree and more, on trees whose CTAs are resident together: 64 trees of depth 5 with 8192 calls 698 us
// against 1882 (a warp per tree), with 256 calls 136 against 195, one tree with 4 calls 107 against 123 and with 1000
// calls 1455 against 9003; 300 trees with 9600 calls 670 against 990, 1000 with 16000 1132 against 1250. Beyond, the
// trees fill the chip by themselves: 4000 with 64000 calls 4654 against 4489; one call each on 1000 trees 165 against 129.
bool trees_set_octants(uint32_t n_trees, uint64_t n_calls, int num_sms) {
    return n_calls >= 4ull * n_trees && n_trees <= 8u * (uint32_t)num_sms;
}

cudaError_t launch_trees_set(const DevInterner &I, const SetCalls &c, uint64_t *list, unsigned long long fc0,
                             unsigned long long ni0, uint32_t *frontier_a, uint32_t *frontier_b, int max_depth,
                             int num_sms, cudaStream_t s) {
    unsigned g = c.n_groups;  // one-warp CTAs: few trees spread over the SMs
    if (g > (unsigned)num_sms * 16) g = (unsigned)num_sms * 16;
    if (g == 0) g = 1;
    count_launches(1);
    if (c.results)
        trees_set_octants_kernel<<<c.n_groups, kOctantThreads, 0, s>>>(I, c);
    else
        trees_set_kernel<<<g, 32, 0, s>>>(I, c);
    cudaError_t e = launch_epoch_refcounts(I, num_sms, s);
    if (e != cudaSuccess) return e;
    unsigned gr = (c.n_groups + kThreads - 1) / kThreads;
    count_launches(2);
    trees_set_roots_kernel<<<gr ? gr : 1, kThreads, 0, s>>>(I, c, list);
    trees_set_garbage_kernel<<<(unsigned)num_sms * 4, kThreads, 0, s>>>(I, fc0, ni0, list);
    return launch_release(I, list, frontier_a, frontier_b, max_depth + 2, num_sms, s);
}

cudaError_t launch_tree_fill(const DevInterner &I, uint32_t tree, uint32_t v, uint64_t *queue, uint64_t queue_cap,
                             HostReply *r, cudaStream_t s) {
    count_launches(1);
    tree_fill_kernel<<<1, kFillThreads, 0, s>>>(I, tree, v, queue, queue_cap, r);
    return cudaGetLastError();
}

cudaError_t launch_rehash(const DevInterner &I, uint64_t table_slots, int num_sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(I.table, 0xFF, table_slots * sizeof(uint64_t), s);
    if (e != cudaSuccess) return e;
    count_launches(1);
    rehash_kernel<<<num_sms * 4, kThreads, 0, s>>>(I);
    count_launches(1);
    rehash_done_kernel<<<1, 1, 0, s>>>(I);
    return cudaGetLastError();
}

cudaError_t launch_reset(const DevInterner &I, int num_sms, cudaStream_t s) {
    count_launches(1);
    reset_kernel<<<num_sms * 8, kThreads, 0, s>>>(I);
    return cudaGetLastError();
}

cudaError_t launch_count_live(const DevInterner &I, unsigned long long *out2, int num_sms, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out2, 0, 2 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    count_launches(1);
    count_live_kernel<<<num_sms * 4, kThreads, 0, s>>>(I, out2);
    return cudaGetLastError();
}

}  // namespace vxg
