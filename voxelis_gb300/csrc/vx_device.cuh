// Device-side data structures and primitives of the GB300 interner.
//
// The interner (the reference's VoxInterner<T>, interner/mod.rs:25-40) lives in HBM as SoA arrays
// of `capacity` node records (capacity = budget / node_size, interner/mod.rs:49-53, 158-164):
//   children[8*i]  u64 BlockIds of the 8 children (zero for leaves)      64 B
//   values[i]      u8 / u16 voxel value (leaf) or LOD value (branch)      1-2 B
//   refcount[i]    u32                                                     4 B
//   generation[i]  u16, bumped when the slot is recycled                  2 B
//   hash[i]        u64 key fingerprint (branches)                          8 B
//   ids[i]         u64 live BlockId of the slot, 0 while free            (+8 B, outside the budget)
// Hash-consing tables (outside the budget, like the reference's HashMaps):
//   table[]        open-addressed branch table of 64-bit slots: tag (32 bits of the key
//                  fingerprint) | node index. Inserts claim a slot with atomicCAS and publish the
//                  index after writing the node; lookups compare the full key (types, mask and the
//                  8 child ids), so equal keys always dedup and unequal keys never alias.
//   leaf_table[v]  direct-mapped leaf ids, one slot per voxel value (0 = none, 1 = being created).
// Allocation pops the LIFO free list first, then bumps next_index (interner/macros.rs:1-41).
// Every spin-wait is bounded; failures set sticky error bits that the host turns into statuses.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace vxg {

constexpr uint64_t EMPTY_ID = 0ull;
constexpr uint64_t INVALID_ID = ~0ull;
constexpr uint16_t MAX_GENERATION = 0x7FFE;
constexpr uint32_t NO_NODE = 0xFFFFFFFFu;

// table slot encoding
constexpr uint64_t SLOT_EMPTY = ~0ull;
constexpr uint64_t SLOT_TOMB = 0xFFFFFFFEFFFFFFFEull;
constexpr uint32_t IDX_BUSY = 0xFFFFFFFFu;
constexpr uint64_t LEAF_BUSY = 1ull;

// sticky error bits (mapped to VX_E_* by the host)
enum : uint32_t {
    ERR_OOM = 1u << 0,
    ERR_TABLE_FULL = 1u << 1,
    ERR_TIMEOUT = 1u << 2,
    ERR_REF_PANIC = 1u << 3,
    ERR_REF_UB = 1u << 4,
    ERR_OOB = 1u << 5,
    ERR_INTERNAL = 1u << 6,
    ERR_INVALID = 1u << 7,
};

constexpr uint8_t TREE_UNUSED = 0xFF;  // depth marker of a free tree slot

// Bounds of every wait. The copy waits of the dense kernels (TMA tiles, and the drain of a warp's
// own copies after giving up) always use SPIN_LIMIT; the waits on other threads (leaf creation, grid
// barriers) use the interner's spin_limit and the warp-intern loop its round_limit,
// both settable per interner (vx_interner_set_limits) and SPIN_LIMIT / ROUND_LIMIT by default.
constexpr uint32_t SPIN_LIMIT = 1u << 22;   // bounded waits (~tens of ms with nanosleep)
constexpr uint32_t ROUND_LIMIT = 1u << 20;  // bounded warp-intern rounds

// DevCounters::alloc_count: the epoch's tickets in the low bits, in the others the tombstones its inserts
// took, so that counting those costs an insert no second atomic on the line every insert goes to.
constexpr int kTicketBits = 33;  // more than the largest capacity (32 bits) twice over
constexpr unsigned long long kTicketMask = (1ull << kTicketBits) - 1ull;

struct DevCounters {
    unsigned long long next_index;   // bump pointer
    unsigned long long free_count;   // free-list length
    unsigned long long alloc_count;  // allocations in the current epoch (kTicketBits), reused tombstones above
    unsigned long long tombstones;   // deleted branch-table slots
    unsigned int error;              // sticky ERR_* bits
    unsigned int error_info;         // first error detail
    unsigned long long scratch[10];  // per-launch counters used by the kernels
    unsigned long long created;      // nodes allocated since the interner was created or reset
    unsigned long long bar_count;    // grid barrier of single-launch kernels: arrivals, only growing
    unsigned long long bar_gen;      //   and their number when the next launch starts
    unsigned long long rel_count[3]; // dying-set sizes of release rounds (rotating; zero between launches)
};

struct DevInterner {
    uint64_t *children;
    void *values;
    uint32_t *refcount;
    uint16_t *generation;
    uint64_t *hash;
    uint64_t *ids;
    uint32_t *free_list;
    DevCounters *ctr;
    uint64_t *table;
    uint64_t table_mask;
    uint64_t *leaf_table;
    uint64_t *roots;
    uint8_t *depths;
    uint32_t tree_cap;
    uint32_t capacity;
    int vbits;
    uint32_t flags;
    uint32_t max_probes;   // branch-table probes before ERR_TABLE_FULL
    uint32_t round_limit;  // warp-intern rounds before ERR_TIMEOUT
    uint32_t spin_limit;   // iterations of a wait on another thread before ERR_TIMEOUT
    uint32_t memo_shift;   // dense builds: quad-memo slots ~ the call's quads >> memo_shift (tunable)
};

// ---- BlockId (core/block_id.rs:19-418) -------------------------------------------------------
__host__ __device__ __forceinline__ bool id_is_leaf(uint64_t id) { return (id >> 63) != 0; }
__host__ __device__ __forceinline__ bool id_is_branch(uint64_t id) { return (id >> 63) == 0; }
__host__ __device__ __forceinline__ uint32_t id_index(uint64_t id) { return (uint32_t)id; }
__host__ __device__ __forceinline__ uint32_t id_generation(uint64_t id) { return (uint32_t)((id >> 32) & 0x7FFF); }
__host__ __device__ __forceinline__ uint32_t id_types(uint64_t id) { return (uint32_t)((id >> 55) & 0xFF); }
__host__ __device__ __forceinline__ uint32_t id_mask(uint64_t id) { return (uint32_t)((id >> 47) & 0xFF); }
__host__ __device__ __forceinline__ uint64_t make_leaf_id(uint32_t index, uint32_t gen) {
    return (1ull << 63) | ((uint64_t)(gen & 0x7FFF) << 32) | index;
}
__host__ __device__ __forceinline__ uint64_t make_branch_id(uint32_t index, uint32_t gen, uint32_t types,
                                                            uint32_t mask) {
    return ((uint64_t)(types & 0xFF) << 55) | ((uint64_t)(mask & 0xFF) << 47) |
           ((uint64_t)(gen & 0x7FFF) << 32) | index;
}

// ---- memory helpers --------------------------------------------------------------------------
__device__ __forceinline__ uint64_t ld_volatile(const uint64_t *p) { return *(const volatile uint64_t *)p; }
// Acquire load of a table slot: the node record published before the slot is visible after it.
__device__ __forceinline__ uint64_t ld_acquire(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t ld_cg(const uint64_t *p) { return __ldcg((const unsigned long long *)p); }
// Load of a hash-table slot while probing: what its publisher wrote before it is visible after it. (An acquire
// costs nothing against a relaxed load on 500 to 190 000 bottom groups, 2 % on 6.3 M.)
__device__ __forceinline__ uint64_t ld_probe(const uint64_t *p) { return ld_acquire(p); }
// The same of a 32-byte sector of four slots.
__device__ __forceinline__ void ld_probe_sector(const uint64_t *p, uint64_t w[4]) {
    asm volatile("ld.acquire.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ void ld_relaxed_sector(const uint64_t *p, uint64_t w[4]) {
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Publication with release semantics: every store of this thread before it is visible to a thread
// that reads the new value with acquire semantics (ld_probe). Cheaper than a full fence before a
// plain atomic, which also orders loads and waits for sequential consistency.
__device__ __forceinline__ unsigned long long atom_exch_release(unsigned long long *p, unsigned long long v) {
    unsigned long long old;
    asm volatile("atom.release.gpu.global.exch.b64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
    return old;
}
// Publication of a slot this thread owns (claimed in a busy state that no other thread writes): a
// release store waits for this thread's earlier writes like the exchange, but not for a reply.
#ifndef VX_PUB_STORE
#define VX_PUB_STORE 1
#endif
__device__ __forceinline__ void publish_release(unsigned long long *p, unsigned long long v) {
    if (VX_PUB_STORE)
        st_release_u64(p, v);
    else
        atom_exch_release(p, v);
}
// Compare-and-swap that publishes this thread's earlier stores (release) and, whatever its outcome,
// makes the stores published with the value it read visible to this thread (acquire).
__device__ __forceinline__ unsigned long long atom_cas_acq_rel(unsigned long long *p, unsigned long long cmp,
                                                               unsigned long long v) {
    unsigned long long old;
    asm volatile("atom.acq_rel.gpu.global.cas.b64 %0, [%1], %2, %3;" : "=l"(old) : "l"(p), "l"(cmp), "l"(v) : "memory");
    return old;
}

// Counts the calling CTA as done on *done and returns true in thread 0 of the last CTA of the grid to
// finish (every other CTA's writes are visible to it), after resetting *done for the next kernel.
// All threads of the CTA must call it. Lets a kernel's last CTA do the one-thread follow-up work that
// would otherwise be a separate launch.
__device__ __forceinline__ bool grid_last_cta(unsigned long long *done) {
    __shared__ unsigned int is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = atomicAdd(done, 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (threadIdx.x != 0 || !is_last) return false;
    __threadfence();
    *done = 0;
    return true;
}

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute may
// start while its predecessor on the stream still runs; pdl_wait() blocks until the predecessor has
// completed and its writes are visible (a no-op for a normal launch), and pdl_release() lets the next
// kernel of the stream launch early. A kernel calls pdl_wait() before its first access to memory the
// predecessor writes.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void set_error(const DevInterner &I, uint32_t bit, uint32_t info = 0) {
    unsigned int old = atomicOr(&I.ctr->error, bit);
    if (old == 0) atomicExch(&I.ctr->error_info, info);
}

__device__ __forceinline__ uint32_t node_value(const DevInterner &I, uint32_t idx) {
    return I.vbits == 8 ? (uint32_t)((const uint8_t *)I.values)[idx] : (uint32_t)((const uint16_t *)I.values)[idx];
}
__device__ __forceinline__ uint32_t node_value_cg(const DevInterner &I, uint32_t idx) {
    if (I.vbits == 8) return (uint32_t)__ldcg((const unsigned char *)I.values + idx);
    return (uint32_t)__ldcg((const unsigned short *)I.values + idx);
}
__device__ __forceinline__ void set_node_value(const DevInterner &I, uint32_t idx, uint32_t v) {
    if (I.vbits == 8)
        ((uint8_t *)I.values)[idx] = (uint8_t)v;
    else
        ((uint16_t *)I.values)[idx] = (uint16_t)v;
}

// ---- key fingerprint -------------------------------------------------------------------------
__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}
__device__ __forceinline__ uint64_t branch_fingerprint(const uint64_t c[8], uint32_t tm) {
    uint64_t h = 0x9E3779B97F4A7C15ull ^ ((uint64_t)tm << 17);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h ^= c[i] * 0x87C37B91114253D5ull;
        h = ((h << 31) | (h >> 33)) * 0x4CF5AD432745937Full;
    }
    return fmix64(h);
}
__device__ __forceinline__ uint32_t slot_tag(uint64_t h) {
    uint32_t t = (uint32_t)(h >> 32);
    return t >= 0xFFFFFFFEu ? 0xFFFFFFFDu : t;
}
__device__ __forceinline__ uint64_t make_slot(uint32_t tag, uint32_t idx) { return ((uint64_t)tag << 32) | idx; }

// calc_average (core/voxel.rs:96-141): the mode of the 8 values. Distinct values are visited in
// first-seen order; a later value replaces the current best when it is more frequent, or equally
// frequent while the best is the default value and it is not. So the result is the first value other than
// the default that is as frequent as any, or the default when none is. Each of the 28 pairs is compared
// once, fully unrolled on registers.
__device__ __forceinline__ uint32_t calc_average8(const uint32_t v[8]) {
    uint32_t cnt[8] = {1, 1, 1, 1, 1, 1, 1, 1};
#pragma unroll
    for (int k = 1; k < 8; ++k)
#pragma unroll
        for (int j = 0; j < k; ++j) {
            const uint32_t same = v[j] == v[k] ? 1u : 0u;
            cnt[j] += same;
            cnt[k] += same;
        }
    uint32_t most = cnt[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) most = max(most, cnt[k]);
    uint32_t best = 0;
#pragma unroll
    for (int k = 7; k >= 0; --k) best = (cnt[k] == most && v[k] != 0) ? v[k] : best;
    return best;
}

// ---- allocation --------------------------------------------------------------------------------
// The t-th allocation of an epoch takes free_list[free_count-1-t] while the free list lasts, then
// next_index + (t - free_count). free_count and next_index only change between epochs.
__device__ __forceinline__ uint32_t node_for_ticket(const DevInterner &I, unsigned long long t,
                                                    unsigned long long fc, unsigned long long ni) {
    unsigned long long idx = (t < fc) ? (unsigned long long)I.free_list[fc - 1 - t] : ni + (t - fc);
    return idx < I.capacity ? (uint32_t)idx : NO_NODE;
}
__device__ __forceinline__ uint32_t node_for_ticket(const DevInterner &I, unsigned long long t) {
    return node_for_ticket(I, t, I.ctr->free_count, I.ctr->next_index);
}

// Closes the epoch (one thread, after every allocation of the epoch): the free-list entries and
// fresh indices its tickets took become allocated.
__device__ __forceinline__ void epoch_finalize_body(const DevInterner &I) {
    DevCounters *c = I.ctr;
    const unsigned long long alloc = c->alloc_count & kTicketMask, fc = c->free_count;
    c->tombstones -= c->alloc_count >> kTicketBits;
    const unsigned long long used_free = alloc < fc ? alloc : fc;
    c->free_count = fc - used_free;
    unsigned long long ni = c->next_index + (alloc - used_free);
    if (ni > I.capacity) ni = I.capacity;
    c->created += used_free + (ni - c->next_index);
    c->next_index = ni;
    c->alloc_count = 0;
}

// Slots past next_index have never held a node since the interner was created or reset (the bump
// allocator hands each out once, recycling only bumps the generation of slots handed out before,
// and creation, reset and model loading zero the generations), so their generation is 0: a ticket
// past the free list needs no dependent load of it.
#ifndef VX_FRESH_GEN
#define VX_FRESH_GEN 1
#endif
__device__ __forceinline__ uint32_t slot_generation(const DevInterner &I, uint32_t idx, bool bumped) {
    return (VX_FRESH_GEN && bumped) ? 0u : (uint32_t)I.generation[idx];
}

// Writes a new branch record (children, LOD value, fingerprint, live id); rc starts at 0. bumped: idx
// came from past the free list (generation 0).
__device__ __forceinline__ uint64_t write_branch(const DevInterner &I, uint32_t idx, const uint64_t c[8],
                                                 uint32_t types, uint32_t mask, uint64_t h, uint32_t lod,
                                                 bool bumped = false) {
    uint32_t gen = slot_generation(I, idx, bumped);
    uint64_t id = make_branch_id(idx, gen, types, mask);
    ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(I.children + 8ull * idx);
    dst[0] = make_ulonglong2(c[0], c[1]);
    dst[1] = make_ulonglong2(c[2], c[3]);
    dst[2] = make_ulonglong2(c[4], c[5]);
    dst[3] = make_ulonglong2(c[6], c[7]);
    set_node_value(I, idx, lod);
    I.hash[idx] = h;
    I.refcount[idx] = 0;
    I.ids[idx] = id;
    return id;
}

// The id and the children of node idx are loaded together (one round trip); *id_out gets the id.
__device__ __forceinline__ bool key_equal(const DevInterner &I, uint32_t idx, const uint64_t c[8], uint32_t types,
                                          uint32_t mask, uint64_t *id_out = nullptr) {
    const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * idx);
    const uint64_t id = ld_cg(I.ids + idx);
    ulonglong2 w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = __ldcg(src + k);
    if (id == 0 || id_is_leaf(id) || id_types(id) != types || id_mask(id) != mask) return false;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (w[k].x != c[2 * k] || w[k].y != c[2 * k + 1]) return false;
    if (id_out) *id_out = id;
    return true;
}

// The rest of the 32-byte sector of slot `pos` in one load (a miss brings the sector anyway, and the warp steps at
// the pace of its longest probe sequence; 6.3 M bottom groups and their undo 5.97 ms, 6.17 a slot at a time): moves pos and probes to the first slot that is
// EMPTY or has the tag and returns it, noting the first tombstone on the way; SLOT_TOMB when there is none
// (pos and probes are then past the sector, or past the probe limit).
__device__ __forceinline__ uint64_t probe_sector(const DevInterner &I, uint32_t tag, uint64_t &pos, uint32_t &probes,
                                                 uint32_t &tomb) {
    uint64_t w[4];
    ld_probe_sector(I.table + (pos & ~3ull), w);
    const uint32_t j = (uint32_t)pos & 3u, top = (uint32_t)I.table_mask & 3u;  // (tables of 2 slots)
    uint64_t s = SLOT_TOMB;
    uint32_t at = top + 1u;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        if (k < j || k >= at) continue;
        if (w[k] == SLOT_TOMB) {
            if (tomb == 0) tomb = probes + (k - j) + 1u;
        } else if (w[k] == SLOT_EMPTY || (uint32_t)(w[k] >> 32) == tag) {
            s = w[k];
            at = k;
        }
    }
    pos = (pos + (at - j)) & I.table_mask;
    probes += at - j;
    return probes > I.max_probes ? SLOT_TOMB : s;
}

// Warp-cooperative find-or-insert of branch keys. Every lane of the warp must call it (converged);
// lanes with active == false only take part in the ballots. Each round every unfinished lane makes
// one non-blocking probe step; a lane that claimed a slot waits until no lane of the warp can step on
// (all have claimed, finished, or met a slot still being written), and then all of them take node indices
// from a single ticket range, write their nodes and publish them. A lane that meets a slot still being
// written retries it next round, so no lane ever waits inside a divergent branch, and a warp never waits
// while it holds a claim. The tickets bound this: one counter for the whole grid, and behind it a chain of
// the reply, the free list, the generation and the fence of the publication. Taken after each round with a
// claim, 3 to 6 times a warp, it made an apply of 6.3 M bottom groups and its undo 7.5 ms; taken once 6.4.
// A new key takes the first tombstone of its probe sequence, once the sequence has reached an EMPTY slot
// without meeting the key. Slots only go from EMPTY or tombstone to a key while nodes are created, so two
// lanes with one key agree on the slot or one of them loses the compare-and-swap, and a loser goes on from
// the slot it lost. Edits that come and go recreate the same keys (the bottom groups of a fill and its
// undo): without reuse each left one more tombstone for its next insert to walk over, and 4096 edits of a
// 512^3 tree and their undo grew from 1.9 to 8.0 ms a pass before the table was rebuilt.
// Returns the BlockId; *created tells whether this lane inserted the node. On failure (probe limit,
// round limit, out of nodes: a sticky error bit is set) the lane gets EMPTY_ID, which every consumer
// handles without dereferencing it, so a failed call leaves wrong but memory-safe results until
// vx_interner_reset.
#ifndef VX_INTERN_INLINE
#define VX_INTERN_INLINE __noinline__
#endif
// lod_of() gives the LOD value of a new node. It is called once, behind the first probe, so that a caller whose
// children's values are still on their way does not wait for them before it (an apply of 261 K records of a tree of
// depth 9 577 us against 588, of 16 K 363 against 373).
template <class Lod>
__device__ __forceinline__ uint64_t warp_intern_branch_inl(const DevInterner &I, bool active, const uint64_t c[8],
                                                           uint32_t types, uint32_t mask, Lod lod_of, bool *created,
                                                           uint64_t h_in = 0) {
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t tm = (types << 8) | mask;
    uint64_t h = 0;
    uint32_t tag = 0;
    uint64_t pos = 0;
    uint32_t probes = 0;
    uint32_t tomb = 0;  // 1 + probes before the first tombstone met, 0: none
    bool done = !active;
    uint64_t result = EMPTY_ID;
    *created = false;
    // constant during an epoch: loaded beside the first probe instead of after a ticket is taken
    const unsigned long long fc = I.ctr->free_count, ni = I.ctr->next_index;
    if (active) {
        h = h_in ? h_in : branch_fingerprint(c, tm);
        tag = slot_tag(h);
        pos = h & I.table_mask;
    }
    bool claimed = false;
    uint32_t lod = 0;
    for (uint32_t round = 0;; ++round) {
        bool waiting = false;
        if (!done && !claimed) {
            uint64_t s = probe_sector(I, tag, pos, probes, tomb);
            if (s == SLOT_EMPTY) {
                if (tomb) {
                    probes = tomb - 1;
                    pos = (h + probes) & I.table_mask;
                }
                const uint64_t free_slot = tomb ? SLOT_TOMB : SLOT_EMPTY;
                uint64_t prev = atomicCAS((unsigned long long *)(I.table + pos), free_slot, make_slot(tag, IDX_BUSY));
                if (prev == free_slot) {
                    claimed = true;
                } else {
                    s = prev;
                    tomb = 0;
                }
            }
            if (!claimed) {
                if ((uint32_t)(s >> 32) == tag && s != SLOT_TOMB) {
                    uint32_t idx = (uint32_t)s;
                    if (idx == IDX_BUSY) {
                        waiting = true;  // retry the same slot next round
                    } else if (key_equal(I, idx, c, types, mask, &result)) {
                        done = true;
                    } else {
                        pos = (pos + 1) & I.table_mask;
                        ++probes;
                    }
                } else if (s != SLOT_TOMB) {  // lost a slot to another key
                    pos = (pos + 1) & I.table_mask;
                    ++probes;
                }
                if (!done && probes > I.max_probes) {
                    set_error(I, ERR_TABLE_FULL, 1);
                    done = true;
                }
            }
        }
        if (round == 0) lod = lod_of();
        const bool last = round >= I.round_limit;
        const unsigned cm = __ballot_sync(0xFFFFFFFFu, claimed);
        if (cm && (last || !__any_sync(0xFFFFFFFFu, !done && !claimed && !waiting))) {
            unsigned long long base = 0;
            const int leader = __ffs(cm) - 1;
            const unsigned reused = __ballot_sync(0xFFFFFFFFu, claimed && tomb != 0);
            if ((int)lane == leader)
                base = atomicAdd(&I.ctr->alloc_count,
                                 (unsigned long long)__popc(cm) | ((unsigned long long)__popc(reused) << kTicketBits));
            base = __shfl_sync(0xFFFFFFFFu, base & kTicketMask, leader);
            if (claimed) {
                const unsigned rank = __popc(cm & ((1u << lane) - 1u));
                const uint32_t idx = node_for_ticket(I, base + rank, fc, ni);
                if (idx == NO_NODE) {
                    set_error(I, ERR_OOM, 1);
                    atomicExch((unsigned long long *)(I.table + pos), SLOT_TOMB);
                    if (tomb) atomicAdd(&I.ctr->tombstones, 1ull);
                } else {
                    result = write_branch(I, idx, c, types, mask, h, lod, base + rank >= fc);
                    publish_release((unsigned long long *)(I.table + pos), make_slot(tag, idx));
                    *created = true;
                }
                claimed = false;
                done = true;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, !done)) break;
        if (last) {
            if (!done) {
                set_error(I, ERR_TIMEOUT, 2);
                done = true;
            }
            break;
        }
        if (waiting) __nanosleep(32);
    }
    return result;
}

// The same, out of line (for call sites on rare paths, to keep kernels small).
static __device__ VX_INTERN_INLINE uint64_t warp_intern_branch(const DevInterner &I, bool active, const uint64_t c[8],
                                                       uint32_t types, uint32_t mask, uint32_t lod, bool *created,
                                                       uint64_t h_in = 0) {
    return warp_intern_branch_inl(I, active, c, types, mask, [=] { return lod; }, created, h_in);
}

// Find-or-create of the leaf for value v (v != 0) through the direct-mapped leaf table.
// *created tells whether this call allocated the leaf (its refcount starts at 0). On failure (out of
// nodes, wait limit: sticky error bit set) it returns EMPTY_ID, like warp_intern_branch.
__device__ __forceinline__ uint64_t intern_leaf(const DevInterner &I, uint32_t v, bool *created) {
    *created = false;
    unsigned long long *slot = (unsigned long long *)(I.leaf_table + v);
    uint64_t s = ld_volatile(I.leaf_table + v);
    if (s > LEAF_BUSY) return s;
    // constant during an epoch: loaded before the claim instead of after the ticket
    const unsigned long long fc = I.ctr->free_count, ni = I.ctr->next_index;
    for (uint32_t spin = 0; spin < I.spin_limit; ++spin) {
        if (s == 0) {  // free (or its creator ran out of memory and backed off): claim it
            const uint64_t prev = atomicCAS(slot, 0ull, LEAF_BUSY);
            if (prev == 0) {
                const unsigned long long t = atomicAdd(&I.ctr->alloc_count, 1ull) & kTicketMask;
                const uint32_t idx = node_for_ticket(I, t, fc, ni);
                if (idx == NO_NODE) {
                    set_error(I, ERR_OOM, 2);
                    atomicExch(slot, 0ull);
                    return EMPTY_ID;
                }
                const uint64_t id = make_leaf_id(idx, slot_generation(I, idx, t >= fc));
                set_node_value(I, idx, v);
                I.hash[idx] = 0;
                I.refcount[idx] = 0;
                I.ids[idx] = id;
                publish_release(slot, id);
                *created = true;
                return id;
            }
            if (prev > LEAF_BUSY) return prev;
        }
        __nanosleep(64);  // being created by another thread
        s = ld_volatile(I.leaf_table + v);
        if (s > LEAF_BUSY) return s;
    }
    set_error(I, ERR_TIMEOUT, 3);
    return EMPTY_ID;
}

// Removes a dead node (id: its BlockId, h: its fingerprint, gen: its generation) from its table, clears the
// record, bumps the generation and puts the slot on the free list at `free_pos` (recycle,
// interner/mod.rs:566-625). A branch's table slot always becomes a tombstone: freeing it where the next
// slot is EMPTY leaves fewer of them, but the ones that stay then sit in runs that end in a live key,
// every insert that hashes into a run lengthens it, and the rebuild that would end it comes late (edits of
// a 512^3 tree: 1.4 ms an apply growing to 6 ms over 150 applies).
__device__ __forceinline__ void recycle_node(const DevInterner &I, uint32_t idx, uint64_t id, uint64_t h, uint32_t gen,
                                             unsigned long long free_pos) {
    if (id_is_leaf(id)) {
        uint32_t v = node_value(I, idx);
        atomicCAS((unsigned long long *)(I.leaf_table + v), id, 0ull);
    } else {
        const uint64_t slot = make_slot(slot_tag(h), idx);
        // a 32-byte sector of four slots a load, as probe_sector
        const uint32_t top = (uint32_t)I.table_mask & 3u;  // (tables of 2 slots)
        uint64_t pos = h & I.table_mask;
        bool removed = false, end = false;
        for (uint32_t p = 0; p <= I.max_probes && !removed && !end;) {
            uint64_t w[4];
            ld_relaxed_sector(I.table + (pos & ~3ull), w);
            const uint32_t j = (uint32_t)pos & 3u;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                if (k < j || k > top || removed || end) continue;
                end = w[k] == SLOT_EMPTY;
                if (w[k] == slot) {  // nothing else writes a published slot while nodes are released
                    *(volatile uint64_t *)(I.table + (pos & ~3ull) + k) = SLOT_TOMB;
                    removed = true;
                }
            }
            pos = (pos + (top + 1u - j)) & I.table_mask;
            p += top + 1u - j;
        }
        if (!removed) set_error(I, ERR_INTERNAL, 10);
        ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(I.children + 8ull * idx);
        dst[0] = dst[1] = dst[2] = dst[3] = make_ulonglong2(0ull, 0ull);
    }
    set_node_value(I, idx, 0);
    I.hash[idx] = 0;
    I.refcount[idx] = 0;
    I.ids[idx] = 0;
    I.generation[idx] = (uint16_t)(gen + 1u >= MAX_GENERATION ? 0u : gen + 1u);
    I.free_list[free_pos] = idx;
}

// ---- barriers of kernels that run in phases ------------------------------------------------------------
// Barrier of all threads of the launch; writes before it are visible to all after it. sync() returns
// false when its bounded wait gave up (ERR_TIMEOUT recorded).
// Grid: a cooperative launch (every CTA resident). Thread 0 of each CTA adds one to a counter that only
// grows and waits for it to reach the barrier's number of arrivals: one round trip after the last arrival.
// The counter's value at the start of a launch is kept beside it, and moved by the first CTA as it leaves
// (every CTA has read it by then).
struct GridBarrier {
    const DevInterner &I;
    unsigned long long target;
    __device__ explicit GridBarrier(const DevInterner &i) : I(i), target(*(volatile unsigned long long *)&i.ctr->bar_gen) {}
    // After a barrier that gave up the arrivals are out of step until the interner is reset.
    __device__ bool usable() { return !(*reinterpret_cast<volatile unsigned int *>(&I.ctr->error) & ERR_TIMEOUT); }
    __device__ bool sync() {
        __shared__ int ok_s;
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            int ok = 1;
            __threadfence();
            atomicAdd(&I.ctr->bar_count, 1ull);
            for (uint32_t spin = 0; (long long)(ld_acquire(reinterpret_cast<const uint64_t *>(&I.ctr->bar_count)) - target) < 0;) {
                // a CTA that gave up at an earlier barrier never arrives: stop waiting at once
                const bool gave_up = (spin & 1023u) == 1023u &&
                                     (*reinterpret_cast<volatile unsigned int *>(&I.ctr->error) & ERR_TIMEOUT);
                if (++spin >= I.spin_limit || gave_up) {
                    set_error(I, ERR_TIMEOUT, 49);
                    ok = 0;
                    break;
                }
                __nanosleep(20);
            }
            __threadfence();
            ok_s = ok;
        }
        __syncthreads();
        return ok_s != 0;
    }
    __device__ void leave() {
        if (blockIdx.x == 0 && threadIdx.x == 0) I.ctr->bar_gen = target;
    }
};

// ---- release (dec_ref_recursive, interner/mod.rs:419-534, breadth first) ------------------------
// Counter slot of the listed roots' number in DevCounters::scratch (the batched-apply launcher's table
// lists every slot).
constexpr int kScRelease = 3;
// Slot of the free list's length at the start of the release rounds (written before the barrier in front of them).
constexpr int kScFreeBase = 4;
// Slot that says whether the release of an apply's set phase waits for that of its clear pass.
constexpr int kScDefer = 5;

__device__ __forceinline__ void push_dying(uint32_t *list, unsigned long long *count, bool push, uint32_t idx) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, push);
    if (!m) return;
    const unsigned lane = threadIdx.x & 31u;
    unsigned long long base = 0;
    const int leader = __ffs(m) - 1;
    if ((int)lane == leader) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (push) list[base + __popc(m & ((1u << lane) - 1u))] = idx;
}

// Decrements each listed root (count at scratch[kScRelease]); roots whose count reaches zero become
// the first dying set. Entry cta_base + threadIdx.x, then + stride, ...: the loop is uniform across
// the CTA, so the warp votes inside see whole warps.
__device__ __forceinline__ void release_roots_range(const DevInterner &I, const uint64_t *list, uint32_t *out,
                                                    unsigned long long *n_out, uint64_t cta_base, uint64_t stride) {
    const uint64_t n = I.ctr->scratch[kScRelease];
    for (uint64_t base = cta_base; base < n; base += stride) {
        const uint64_t j = base + threadIdx.x;
        bool dies = false;
        uint32_t idx = 0;
        if (j < n) {
            const uint64_t id = list[j];
            if (id != EMPTY_ID) {
                idx = id_index(id);
                const unsigned old = atomicSub(I.refcount + idx, 1u);
                if (old == 0) {
                    atomicAdd(I.refcount + idx, 1u);
                    set_error(I, ERR_REF_UB, 60);
                } else {
                    dies = old == 1;
                }
            }
        }
        push_dying(out, n_out, dies, idx);
    }
}

// Per-CTA counts of the references that leaves lose in a release round (shared memory,
// release_smem bytes): direct-mapped by node index with the owner as a tag; a leaf whose slot another
// one owns goes straight to its global count. A few leaves are children of most bottom groups: one
// returning atomic for each of their references serialised at those few addresses (4.5 ms for the
// release of 3.2 M nodes with their 25 M child references).
struct LeafDrops {
    uint32_t *key;  // node index + 1, 0 = free
    uint32_t *cnt;
    uint32_t slots;  // power of two
};
inline __host__ __device__ uint32_t release_slots(int vbits) { return vbits == 8 ? 512u : 4096u; }
inline __host__ __device__ size_t release_smem(int vbits) { return (size_t)release_slots(vbits) * 8; }

// Every thread of the CTA calls it; mem: release_smem bytes no thread still uses.
__device__ __forceinline__ LeafDrops leaf_drops_init(const DevInterner &I, uint32_t *mem) {
    LeafDrops D;
    D.slots = release_slots(I.vbits);
    D.key = mem;
    D.cnt = mem + D.slots;
    for (uint32_t k = threadIdx.x; k < 2 * D.slots; k += blockDim.x) mem[k] = 0;
    __syncthreads();
    return D;
}

// Counts n lost references of leaf idx; false when its slot is taken (the caller goes to the global count).
__device__ __forceinline__ bool leaf_drop(const LeafDrops &D, uint32_t idx, uint32_t n) {
    const uint32_t s = (idx * 0x9E3779B1u) >> 8 & (D.slots - 1u), key = idx + 1u;
    uint32_t t = *(volatile uint32_t *)(D.key + s);
    if (t == 0) {
        t = atomicCAS(D.key + s, 0u, key);
        if (t == 0) t = key;
    }
    if (t != key) return false;
    atomicAdd(D.cnt + s, n);
    return true;
}

// Takes n references from node idx; true when none is left. More than it has is the reference's
// underflow: the count stays at zero and the error is recorded.
__device__ __forceinline__ bool drop_refs(const DevInterner &I, uint32_t idx, uint32_t n, uint32_t old) {
    if (old < n) {
        atomicAdd(I.refcount + idx, n - old);
        set_error(I, ERR_REF_UB, 61);
    }
    return old == n;
}

// Retires the n dying nodes of `in`: their children lose one reference each (children reaching
// zero are the next dying set, appended to `out` and counted in *n_out) and the nodes are recycled. A thread
// takes a node; the counts of its branch children are decremented together, those of leaves in D, which
// the CTA flushes at the end. Node j of the set goes to place free_base + j of the free list, and one thread
// adds the set to the counters: a place and a count taken by every warp serialise at the two counters (an apply of
// 6.3 M bottom groups and its undo, 3.2 M nodes released by each, 6.17 against 6.38 ms). The whole CTA calls it.
__device__ __forceinline__ void release_round_range(const DevInterner &I, const LeafDrops &D, const uint32_t *in,
                                                    uint32_t *out, uint64_t n, uint64_t free_base,
                                                    unsigned long long *n_out, uint64_t cta_base, uint64_t stride) {
    const unsigned lane = threadIdx.x & 31u;
    if (cta_base >= n) return;
    for (uint64_t base = cta_base; base < n; base += stride) {
        const uint64_t j = base + threadIdx.x;
        const bool in_range = j < n;
        const uint32_t idx = in_range ? in[j] : 0u;
        const uint64_t id = in_range ? I.ids[idx] : 0ull;
        const uint64_t h = in_range ? I.hash[idx] : 0ull;
        const uint32_t gen = in_range ? I.generation[idx] : 0u;
        uint64_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (id != 0 && id_is_branch(id)) {
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(I.children + 8ull * idx);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ulonglong2 w = src[k];
                c[2 * k] = w.x;
                c[2 * k + 1] = w.y;
            }
        }
        uint32_t old[8], cnt[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {  // cnt: references to take now; equal children are taken together
            cnt[k] = c[k] != EMPTY_ID ? 1u : 0u;
            old[k] = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i < k && c[i] == c[k]) cnt[k] = 0;
                if (i > k && c[i] == c[k] && cnt[k]) ++cnt[k];
            }
            if (cnt[k] && id_is_leaf(c[k]) && leaf_drop(D, id_index(c[k]), cnt[k])) cnt[k] = 0;
            if (cnt[k]) old[k] = atomicSub(I.refcount + id_index(c[k]), cnt[k]);
        }
        uint32_t dies = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (cnt[k] && drop_refs(I, id_index(c[k]), cnt[k], old[k])) dies |= 1u << k;
        if (__any_sync(0xFFFFFFFFu, dies != 0)) {  // one range of the next dying set for the warp
            const uint32_t mine = __popc(dies);
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (unsigned)o) incl += y;
            }
            unsigned long long at = 0;
            if (lane == 31) at = atomicAdd(n_out, (unsigned long long)incl);
            at = __shfl_sync(0xFFFFFFFFu, at, 31) + (incl - mine);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if ((dies >> k) & 1u) out[at++] = id_index(c[k]);
        }
        const unsigned leaves = __ballot_sync(0xFFFFFFFFu, in_range && id_is_leaf(id));
        if (lane == 0 && leaves) atomicAdd(&I.ctr->tombstones, 0ull - (unsigned long long)__popc(leaves));
        if (!in_range) continue;
        if (id != 0) {
            recycle_node(I, idx, id, h, gen, free_base + j);
        } else {
            I.free_list[free_base + j] = idx;
            set_error(I, ERR_INTERNAL, 62);
        }
    }
    if (cta_base == 0 && threadIdx.x == 0) {
        I.ctr->free_count = free_base + n;
        atomicAdd(&I.ctr->tombstones, n);
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < D.slots; s += blockDim.x) {  // slots: a multiple of the CTA's warps
        const uint32_t n_ref = D.cnt[s];
        bool dies = false;
        uint32_t idx = 0;
        if (n_ref) {
            idx = D.key[s] - 1u;
            dies = drop_refs(I, idx, n_ref, atomicSub(I.refcount + idx, n_ref));
            D.key[s] = 0;
            D.cnt[s] = 0;
        }
        push_dying(out, n_out, dies, idx);
    }
    __syncthreads();
}

}  // namespace vxg
