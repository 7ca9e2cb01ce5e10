// World-level helpers for the serving loop: a grid of equal-depth chunks addressed by world voxel
// coordinates. Not part of the reference's API; they stage the same Batch contents the reference's
// callers build by hand (Batch::just_set per voxel, core/batch.rs:145-172) and read a world with
// VoxTree::get per chunk (voxtree.rs:145-159).
//
//   vx_stage_spheres    sphere brushes (center, radius, value) applied in order as just_set calls
//                       into one Batch per touched chunk, emitted as compacted touched groups
//                       sorted by (chunk, group) — the input of vx_apply_groups_async.
//   vx_world_get_async  batched get at world coordinates: chunk lookup in the device world table,
//                       then the per-tree descent of get_at_depth (utils/common.rs:122-156).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/voxelis_gb300.h"
#include "vx_launch.h"

using namespace vxg;

namespace vxg {
bool interner_parts(vx_interner *it, DevInterner *dev, cudaStream_t *stream, int *num_sms, uint32_t *flags,
                    bool marks_trees);
void interner_set_error(vx_interner *it, const char *msg);
}  // namespace vxg

namespace {

__host__ __device__ uint32_t morton3(uint32_t x, uint32_t y, uint32_t z) {
    auto split = [](uint32_t v) {
        v &= 0x3FF;
        v = (v | (v << 16)) & 0x30000FF;
        v = (v | (v << 8)) & 0x300F00F;
        v = (v | (v << 4)) & 0x30C30C3;
        v = (v | (v << 2)) & 0x9249249;
        return v;
    };
    return split(x) | (split(y) << 1) | (split(z) << 2);
}

struct GroupRec {
    uint64_t key;  // chunk << 32 | group
    uint8_t set, clear;
    uint16_t vals[8];
};

// Open-addressing map key -> record slot, grown at load 1/2.
struct RecMap {
    std::vector<uint64_t> keys;
    std::vector<uint32_t> slot;
    std::vector<GroupRec> recs;
    uint64_t mask = 0;
    void init(size_t cap) {
        size_t n = 1024;
        while (n < 2 * cap) n <<= 1;
        keys.assign(n, ~0ull);
        slot.assign(n, 0);
        mask = n - 1;
        recs.clear();
    }
    GroupRec &at(uint64_t key) {
        if ((recs.size() + 1) * 2 > keys.size()) grow();
        uint64_t h = (key * 0x9E3779B97F4A7C15ull) >> 20;
        for (;;) {
            const uint64_t i = h & mask;
            if (keys[i] == key) return recs[slot[i]];
            if (keys[i] == ~0ull) {
                keys[i] = key;
                slot[i] = (uint32_t)recs.size();
                GroupRec r{};
                r.key = key;
                recs.push_back(r);
                return recs.back();
            }
            ++h;
        }
    }
    void grow() {
        std::vector<GroupRec> old;
        old.swap(recs);
        init(old.size() * 2 + 16);
        for (auto &r : old) {
            GroupRec &n = at(r.key);
            n = r;
        }
    }
};

// Gets at world coordinates. With old_roots, a chunk whose edit_rank is cut or more (and not
// kNoRank) is read at the root held for it before the wave's apply (see vx_world_hold_async).
constexpr uint32_t kNoRank = 0xFFFFFFFFu;

template <class T>
__global__ void world_get_kernel(DevInterner I, vx_world W, uint64_t n, const int32_t *xyz, uint8_t *found,
                                 T *values, const uint64_t *old_roots, const uint32_t *edit_rank, uint32_t cut) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const int d = W.chunk_depth;
    const int32_t side = 1 << d;
    bool oob = false;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
        const int32_t x = __ldg(xyz + 3 * q), y = __ldg(xyz + 3 * q + 1), z = __ldg(xyz + 3 * q + 2);
        uint32_t val = 0;
        uint8_t f = 0;
        if (x < 0 || y < 0 || z < 0 || x >= W.nx * side || y >= W.ny * side || z >= W.nz * side) {
            oob = true;
        } else {
            const uint32_t chunk = ((uint32_t)(y >> d) * W.nz + (uint32_t)(z >> d)) * W.nx + (uint32_t)(x >> d);
            const uint32_t t = __ldg(W.trees_dev + chunk);
            const int32_t lx = x & (side - 1), ly = y & (side - 1), lz = z & (side - 1);
            uint64_t node = t < I.tree_cap ? I.roots[t] : EMPTY_ID;
            if (old_roots) {
                const uint32_t r = __ldg(edit_rank + chunk);
                if (r != kNoRank && r >= cut) node = __ldg(reinterpret_cast<const unsigned long long *>(old_roots) + chunk);
            }
            int depth = 0;
            while (node != EMPTY_ID) {
                if (depth >= d) {
                    const uint32_t v = node_value(I, id_index(node));
                    if (v) {
                        val = v;
                        f = 1;
                    }
                    break;
                }
                if (id_is_branch(node)) {
                    const int sh = d - depth - 1;
                    const uint32_t ci = ((lx >> sh) & 1) | (((ly >> sh) & 1) << 1) | (((lz >> sh) & 1) << 2);
                    node = __ldg(reinterpret_cast<const unsigned long long *>(I.children) + 8ull * id_index(node) + ci);
                    ++depth;
                } else {
                    val = node_value(I, id_index(node));
                    f = 1;
                    break;
                }
            }
        }
        found[q] = f;
        values[q] = (T)val;
    }
    if (oob) set_error(I, ERR_OOB, 90);
}

// Holds the current root of each listed chunk for the gets of a wave that must not see the wave's
// edits: one more reference on it (VoxInterner::inc_ref, interner/mod.rs:235-260), its id in
// held[k] and old_roots[chunk], the rank of the wave's edit of that chunk in edit_rank[chunk].
__global__ void world_hold_kernel(DevInterner I, vx_world W, uint32_t n, const uint32_t *chunks, const uint32_t *ranks,
                                  uint64_t *held, uint64_t *old_roots, uint32_t *edit_rank) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t c = chunks[k];
    if (c >= (uint32_t)(W.nx * W.ny * W.nz)) {
        set_error(I, ERR_OOB, 91);
        held[k] = EMPTY_ID;
        return;
    }
    const uint32_t t = W.trees_dev[c];
    const uint64_t root = t < I.tree_cap ? I.roots[t] : EMPTY_ID;
    held[k] = root;
    old_roots[c] = root;
    edit_rank[c] = ranks[k];
    if (root != EMPTY_ID) atomicAdd(I.refcount + id_index(root), 1u);
}

// Ends the holds: the listed chunks read their current roots again, and the held ids become the
// list of the release that follows (count in the release slot).
__global__ void world_unhold_kernel(DevInterner I, vx_world W, uint32_t n, const uint32_t *chunks, uint32_t *edit_rank) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) I.ctr->scratch[SC_RELEASE] = n;
    if (k < n && chunks[k] < (uint32_t)(W.nx * W.ny * W.nz)) edit_rank[chunks[k]] = kNoRank;
}

// ---- sphere brushes staged on the device -----------------------------------------------------------------
// One touched chunk of a wave: its sphere, in the chunk's voxel coordinates, and its records' place.
struct SphereItem {
    uint32_t chunk, first, sphere, value;
    int32_t center[3], radius;
};

__device__ __forceinline__ uint32_t compact3(uint32_t v) {  // every third bit
    v &= 0x9249249;
    v = (v | (v >> 2)) & 0x30C30C3;
    v = (v | (v >> 4)) & 0x300F00F;
    v = (v | (v >> 8)) & 0x30000FF;
    return (v | (v >> 16)) & 0x3FF;
}

__device__ __forceinline__ uint64_t square(int32_t v) { return (uint64_t)((int64_t)v * v); }

// Voxels of 2x2x2 group g inside the item's sphere, a bit each.
__device__ __forceinline__ uint32_t group_mask(const SphereItem &S, uint32_t g, uint64_t r2) {
    const int32_t dx = 2 * (int32_t)compact3(g) - S.center[0], dy = 2 * (int32_t)compact3(g >> 1) - S.center[1],
                  dz = 2 * (int32_t)compact3(g >> 2) - S.center[2];
    const uint64_t x2[2] = {square(dx), square(dx + 1)}, y2[2] = {square(dy), square(dy + 1)},
                   z2[2] = {square(dz), square(dz + 1)};
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) m |= (x2[k & 1] + y2[(k >> 1) & 1] + z2[k >> 2] <= r2 ? 1u : 0u) << k;
    return m;
}

// Distance from v to [0, n) along an axis, where the interval starts at v = 0.
__device__ __forceinline__ int32_t axis_gap(int32_t lo, int32_t n) { return lo > 0 ? lo : (lo + n <= 0 ? -(lo + n - 1) : 0); }

constexpr int kStageThreads = 512;

// A CTA an item: its warps share the Morton range of the sphere's box in contiguous parts, count the touched
// groups, and then write their records side by side, in order. 32 groups are a block of 4x4x2 groups; each lane
// asks for one whether the sphere meets it, and the warp goes through those that it does. Bound by the launch and
// the apply behind it; what it saves is the host's hash map and sort (350 us a wave of 11 spheres) and the copies
// of 26 bytes a record: 44 spheres and 20 reads served in 1.66 ms, 3.0 when the host staged.
__global__ void __launch_bounds__(kStageThreads) stage_spheres_kernel(DevInterner I, vx_world W, const SphereItem *items,
                                                                      uint32_t n_items, uint32_t n_records,
                                                                      uint32_t *item_trees, uint32_t *item_chunks,
                                                                      uint32_t *item_ranks, uint32_t *rec_item,
                                                                      uint32_t *rec_group, uint8_t *rec_set,
                                                                      uint8_t *rec_clear, uint4 *rec_vals) {
    __shared__ uint32_t counts[kStageThreads / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = kStageThreads / 32;
    const int32_t last = (1 << (W.chunk_depth - 1)) - 1;  // last group of an axis
    for (uint32_t i = blockIdx.x; i < n_items; i += gridDim.x) {
        const SphereItem S = items[i];
        const uint32_t end = i + 1 < n_items ? items[i + 1].first : n_records;
        const uint64_t r2 = square(S.radius);
        int32_t b0[3], b1[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            b0[k] = max(0, (int32_t)max((int64_t)S.center[k] - S.radius, (int64_t)0) >> 1);
            b1[k] = (int32_t)min(((int64_t)S.center[k] + S.radius) >> 1, (int64_t)last);
        }
        const uint32_t first = morton3(b0[0], b0[1], b0[2]) & ~31u, groups = morton3(b1[0], b1[1], b1[2]) + 1;
        const uint32_t part = ((groups - first + 32 * nw - 1) / (32 * nw)) * 32;
        const uint32_t lo = first + warp * part, hi = lo + part < groups ? lo + part : groups;
        uint32_t at = S.first;
        for (int pass = 0; pass < 2; ++pass) {
            uint32_t n = 0;
            unsigned met = 0;
            for (uint32_t base = lo, many = lo; met || many < hi;) {
                if (!met) {  // the next 32 blocks
                    const uint32_t b = many + 32 * lane;
                    const int32_t bx = 2 * (int32_t)compact3(b) - S.center[0], by = 2 * (int32_t)compact3(b >> 1) - S.center[1],
                                  bz = 2 * (int32_t)compact3(b >> 2) - S.center[2];
                    const uint64_t d2 = square(axis_gap(bx, 8)) + square(axis_gap(by, 8)) + square(axis_gap(bz, 4));
                    met = __ballot_sync(0xFFFFFFFFu, b < hi && d2 <= r2);
                    base = many;
                    many += 1024;
                    continue;
                }
                const uint32_t g = base + 32 * (uint32_t)(__ffs(met) - 1) + lane;
                met &= met - 1;
                const uint32_t m = g < hi ? group_mask(S, g, r2) : 0u;
                const unsigned b = __ballot_sync(0xFFFFFFFFu, m != 0);
                const uint32_t p = at + n + __popc(b & ((1u << lane) - 1u));
                n += __popc(b);
                if (pass == 0 || m == 0 || p >= end) continue;
                const uint32_t v = S.value;
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] = (m >> (2 * k) & 1u ? v : 0u) | (m >> (2 * k + 1) & 1u ? v << 16 : 0u);
                rec_item[p] = i;
                rec_group[p] = g;
                rec_set[p] = (uint8_t)(v ? m : 0u);
                rec_clear[p] = (uint8_t)(v ? 0u : m);
                rec_vals[p] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            if (pass == 1) break;
            if (lane == 0) counts[warp] = n;
            __syncthreads();
            uint32_t all = 0;
            for (unsigned k = 0; k < nw; ++k) {
                if (k < warp) at += counts[k];
                all += counts[k];
            }
            if (threadIdx.x == 0) {
                item_trees[i] = S.chunk < (uint32_t)(W.nx * W.ny * W.nz) ? W.trees_dev[S.chunk] : 0u;
                item_chunks[i] = S.chunk;
                item_ranks[i] = S.sphere;
                if (all != end - S.first) set_error(I, ERR_INTERNAL, 80);  // not what the host counted
            }
            __syncthreads();
        }
    }
}

// Largest s with s * s <= v.
int64_t isqrt(int64_t v) {
    int64_t s = (int64_t)std::sqrt((double)v);
    while (s > 0 && s * s > v) --s;
    while ((s + 1) * (s + 1) <= v) ++s;
    return s;
}

// Touched groups of one sphere by chunk, a row of groups at a time; appends an item for each chunk that has any.
void count_sphere(const vx_world &W, const int32_t c[3], int32_t r, uint32_t sphere, uint32_t value,
                  std::vector<SphereItem> &items, std::vector<uint32_t> &counts) {
    const int d = W.chunk_depth;
    const int32_t size[3] = {W.nx << d, W.ny << d, W.nz << d};
    int32_t lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = (int32_t)std::max<int64_t>(0, (int64_t)c[k] - r);
        hi[k] = (int32_t)std::min<int64_t>(size[k] - 1, (int64_t)c[k] + r);
        if (lo[k] > hi[k]) return;
    }
    const int32_t c0[3] = {lo[0] >> d, lo[1] >> d, lo[2] >> d};
    const int32_t cn[3] = {(hi[0] >> d) - c0[0] + 1, (hi[1] >> d) - c0[1] + 1, (hi[2] >> d) - c0[2] + 1};
    counts.assign((size_t)cn[0] * cn[1] * cn[2], 0);
    const auto nearest = [](int32_t g, int32_t lo_k, int32_t hi_k, int32_t ck) {  // of the group's two voxels inside the box
        const int64_t a = std::max(g, lo_k), b = std::min(g + 1, hi_k);
        const int64_t q = std::max<int64_t>(a, std::min<int64_t>(b, ck)) - ck;
        return q * q;
    };
    for (int32_t y = lo[1] & ~1; y <= hi[1]; y += 2)
        for (int32_t z = lo[2] & ~1; z <= hi[2]; z += 2) {
            const int64_t rest = (int64_t)r * r - nearest(y, lo[1], hi[1], c[1]) - nearest(z, lo[2], hi[2], c[2]);
            if (rest < 0) continue;
            const int64_t half = isqrt(rest);
            const int64_t x0 = std::max<int64_t>(lo[0], c[0] - half), x1 = std::min<int64_t>(hi[0], c[0] + half);
            if (x0 > x1) continue;
            uint32_t *row = counts.data() + ((size_t)((y >> d) - c0[1]) * cn[2] + ((z >> d) - c0[2])) * cn[0];
            for (int64_t k = x0 >> d; k <= x1 >> d; ++k)
                row[k - c0[0]] += (uint32_t)((std::min(x1, ((k + 1) << d) - 1) >> 1) - (std::max(x0, k << d) >> 1) + 1);
        }
    for (int32_t y = 0; y < cn[1]; ++y)
        for (int32_t z = 0; z < cn[2]; ++z)
            for (int32_t x = 0; x < cn[0]; ++x) {
                const uint32_t n = counts[((size_t)y * cn[2] + z) * cn[0] + x];
                if (n == 0) continue;
                const int32_t q[3] = {c0[0] + x, c0[1] + y, c0[2] + z};
                SphereItem S;
                S.chunk = ((uint32_t)q[1] * W.nz + (uint32_t)q[2]) * W.nx + (uint32_t)q[0];
                S.first = n;  // its count until the items are in order
                S.sphere = sphere;
                S.value = value;
                for (int k = 0; k < 3; ++k) S.center[k] = c[k] - (q[k] << d);
                S.radius = r;
                items.push_back(S);
            }
}

}  // namespace

extern "C" int vx_stage_spheres(int chunk_depth, int32_t nx, int32_t ny, int32_t nz, uint32_t n,
                                const int32_t *centers, const int32_t *radii, const uint32_t *values,
                                uint64_t cap_items, uint32_t *item_chunks, uint64_t cap_records, uint32_t *rec_item,
                                uint32_t *rec_group, uint8_t *rec_set, uint8_t *rec_clear, uint16_t *rec_vals,
                                uint64_t *n_items, uint64_t *n_records) {
    if (chunk_depth < 1 || chunk_depth > 10 || nx <= 0 || ny <= 0 || nz <= 0 || !n_items || !n_records ||
        (n && (!centers || !radii || !values)))
        return VX_E_INVALID_ARG;
    const int32_t side = 1 << chunk_depth;
    const int32_t WX = nx * side, WY = ny * side, WZ = nz * side;
    RecMap map;
    map.init(4096);
    for (uint32_t s = 0; s < n; ++s) {
        const int32_t cx = centers[3 * s], cy = centers[3 * s + 1], cz = centers[3 * s + 2], r = radii[s];
        const uint32_t v = values[s];
        if (r < 0 || v > 0xFFFF) return VX_E_INVALID_ARG;
        const int32_t x0 = std::max(0, cx - r) & ~1, x1 = std::min(WX - 1, cx + r);
        const int32_t y0 = std::max(0, cy - r) & ~1, y1 = std::min(WY - 1, cy + r);
        const int32_t z0 = std::max(0, cz - r) & ~1, z1 = std::min(WZ - 1, cz + r);
        const int64_t r2 = (int64_t)r * r;
        for (int32_t gy = y0; gy <= y1; gy += 2)
            for (int32_t gz = z0; gz <= z1; gz += 2)
                for (int32_t gx = x0; gx <= x1; gx += 2) {
                    GroupRec *rec = nullptr;
                    for (int k = 0; k < 8; ++k) {
                        const int32_t x = gx + (k & 1), y = gy + ((k >> 1) & 1), z = gz + (k >> 2);
                        if (x > x1 || y > y1 || z > z1 || x < std::max(0, cx - r) || y < std::max(0, cy - r) ||
                            z < std::max(0, cz - r))
                            continue;
                        const int64_t dx = x - cx, dy = y - cy, dz = z - cz;
                        if (dx * dx + dy * dy + dz * dz > r2) continue;
                        if (!rec) {
                            const uint32_t chunk = ((uint32_t)(y >> chunk_depth) * nz + (uint32_t)(z >> chunk_depth)) * nx +
                                                   (uint32_t)(x >> chunk_depth);
                            const uint32_t lx = x & (side - 1), ly = y & (side - 1), lz = z & (side - 1);
                            const uint32_t group = morton3(lx, ly, lz) >> 3;
                            rec = &map.at(((uint64_t)chunk << 32) | group);
                        }
                        // just_set (batch.rs:145-172): last write wins, a zero value records a clear
                        const uint8_t bit = (uint8_t)(1u << k);
                        if (v) {
                            rec->set |= bit;
                            rec->clear &= (uint8_t)~bit;
                        } else {
                            rec->set &= (uint8_t)~bit;
                            rec->clear |= bit;
                        }
                        rec->vals[k] = (uint16_t)v;
                    }
                }
    }
    std::vector<uint32_t> order(map.recs.size());
    for (uint32_t i = 0; i < order.size(); ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return map.recs[a].key < map.recs[b].key; });
    uint64_t items = 0;
    uint64_t last_chunk = ~0ull;
    for (uint32_t i : order) {
        const uint64_t ch = map.recs[i].key >> 32;
        if (ch != last_chunk) {
            ++items;
            last_chunk = ch;
        }
    }
    *n_items = items;
    *n_records = order.size();
    if (items > cap_items || order.size() > cap_records) return VX_E_BUFFER;
    if (!order.empty() && (!item_chunks || !rec_item || !rec_group || !rec_set || !rec_clear || !rec_vals))
        return VX_E_INVALID_ARG;
    int64_t item = -1;
    last_chunk = ~0ull;
    for (uint64_t j = 0; j < order.size(); ++j) {
        const GroupRec &g = map.recs[order[j]];
        const uint64_t ch = g.key >> 32;
        if (ch != last_chunk) {
            ++item;
            item_chunks[item] = (uint32_t)ch;
            last_chunk = ch;
        }
        rec_item[j] = (uint32_t)item;
        rec_group[j] = (uint32_t)(g.key & 0xFFFFFFFFu);
        rec_set[j] = g.set;
        rec_clear[j] = g.clear;
        std::memcpy(rec_vals + 8 * j, g.vals, 16);
    }
    return VX_OK;
}

// Deepest chunk that the device stages. A wave from its spheres to the end of its apply, device against host, in
// chunks of depth 5 to 8: one sphere of radius 2 83-97 us against 109-125, of radius 12 92-117 against 191-207, of
// radius 30 126-289 against 1325-1388, eight of radius 8 107-126 against 325-342. The blocks that the device asks
// about grow eightfold a depth where a sphere sits at the middle of its chunk: some 8 us at depth 8, 65 at 9.
constexpr int kStageDepth = 8;

extern "C" int vx_stage_spheres_async(vx_interner *it, const vx_world *world, uint32_t n, const int32_t *centers,
                                      const int32_t *radii, const uint32_t *values, uint64_t cap_items, void *plan_host,
                                      void *plan_dev, uint32_t *item_trees_dev, uint32_t *item_chunks_dev,
                                      uint32_t *item_ranks_dev, uint64_t cap_records, uint32_t *rec_item_dev,
                                      uint32_t *rec_group_dev, uint8_t *rec_set_dev, uint8_t *rec_clear_dev,
                                      uint16_t *rec_vals_dev, uint64_t *n_items, uint64_t *n_records) try {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false) || !world || !n_items || !n_records ||
        (n && (!centers || !radii || !values)))
        return VX_E_INVALID_ARG;
    const vx_world &W = *world;
    if (W.chunk_depth < 1 || W.chunk_depth > 10 || W.nx <= 0 || W.ny <= 0 || W.nz <= 0 || !W.trees_dev) return VX_E_INVALID_ARG;
    if (W.chunk_depth > kStageDepth) return VX_E_UNSUPPORTED;
    std::vector<SphereItem> items;
    std::vector<uint32_t> counts;
    for (uint32_t k = 0; k < n; ++k) {
        if (radii[k] < 0 || values[k] > 0xFFFF) return VX_E_INVALID_ARG;
        count_sphere(W, centers + 3 * k, radii[k], k, values[k], items, counts);
    }
    std::sort(items.begin(), items.end(), [](const SphereItem &a, const SphereItem &b) { return a.chunk < b.chunk; });
    uint64_t total = 0;
    for (size_t k = 0; k < items.size(); ++k) {
        if (k && items[k].chunk == items[k - 1].chunk) return VX_E_UNSUPPORTED;  // two spheres' records to merge
        const uint32_t c = items[k].first;
        items[k].first = (uint32_t)total;
        total += c;
    }
    *n_items = items.size();
    *n_records = total;
    if (items.size() > cap_items || total > cap_records || total > 0xFFFFFFFFull) return VX_E_BUFFER;
    if (items.empty()) return VX_OK;
    if (!plan_host || !plan_dev || !item_trees_dev || !item_chunks_dev || !item_ranks_dev || !rec_item_dev || !rec_group_dev ||
        !rec_set_dev || !rec_clear_dev || !rec_vals_dev ||
        ((reinterpret_cast<uintptr_t>(rec_vals_dev) | reinterpret_cast<uintptr_t>(plan_dev)) & 15u))
        return VX_E_INVALID_ARG;
    std::memcpy(plan_host, items.data(), items.size() * sizeof(SphereItem));
    cudaError_t e = cudaMemcpyAsync(plan_dev, plan_host, items.size() * sizeof(SphereItem), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        const uint32_t blocks = (uint32_t)std::min<uint64_t>(items.size(), (uint64_t)num_sms * 4);
        count_launches(1);
        stage_spheres_kernel<<<blocks, kStageThreads, 0, s>>>(
            D, W, (const SphereItem *)plan_dev, (uint32_t)items.size(), (uint32_t)total, item_trees_dev, item_chunks_dev,
            item_ranks_dev, rec_item_dev, rec_group_dev, rec_set_dev, rec_clear_dev, (uint4 *)rec_vals_dev);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        interner_set_error(it, cudaGetErrorString(e));
        return VX_E_CUDA;
    }
    return VX_OK;
} catch (const std::bad_alloc &) {
    return VX_E_OOM;
}

extern "C" int vx_world_get_async(vx_interner *it, const vx_world *world, uint64_t n, const int32_t *world_xyz_dev,
                                  uint8_t *found_dev, void *values_dev) {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false) || !world) return VX_E_INVALID_ARG;
    if (n == 0) return VX_OK;
    if (!world->trees_dev || !world_xyz_dev || !found_dev || !values_dev || world->chunk_depth < 0 ||
        world->chunk_depth > 10)
        return VX_E_INVALID_ARG;
    uint64_t blocks = (n + 255) / 256;
    if (blocks > (uint64_t)num_sms * 16) blocks = (uint64_t)num_sms * 16;
    count_launches(1);
    if (D.vbits == 8)
        world_get_kernel<uint8_t><<<(unsigned)blocks, 256, 0, s>>>(D, *world, n, world_xyz_dev, found_dev,
                                                                   (uint8_t *)values_dev, nullptr, nullptr, 0);
    else
        world_get_kernel<uint16_t><<<(unsigned)blocks, 256, 0, s>>>(D, *world, n, world_xyz_dev, found_dev,
                                                                    (uint16_t *)values_dev, nullptr, nullptr, 0);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        interner_set_error(it, cudaGetErrorString(e));
        return VX_E_CUDA;
    }
    return VX_OK;
}

extern "C" int vx_world_hold_async(vx_interner *it, const vx_world *world, uint32_t n, const uint32_t *chunks_dev,
                                   const uint32_t *ranks_dev, uint64_t *held_dev, uint64_t *old_roots_dev,
                                   uint32_t *edit_rank_dev) {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false) || !world) return VX_E_INVALID_ARG;
    if (n == 0) return VX_OK;
    if (!world->trees_dev || !chunks_dev || !ranks_dev || !held_dev || !old_roots_dev || !edit_rank_dev)
        return VX_E_INVALID_ARG;
    count_launches(1);
    world_hold_kernel<<<(n + 255) / 256, 256, 0, s>>>(D, *world, n, chunks_dev, ranks_dev, held_dev, old_roots_dev,
                                                      edit_rank_dev);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        interner_set_error(it, cudaGetErrorString(e));
        return VX_E_CUDA;
    }
    return VX_OK;
}

extern "C" int vx_world_get_at_async(vx_interner *it, const vx_world *world, uint64_t n, const int32_t *world_xyz_dev,
                                     uint8_t *found_dev, void *values_dev, const uint64_t *old_roots_dev,
                                     const uint32_t *edit_rank_dev, uint32_t cut) {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false) || !world) return VX_E_INVALID_ARG;
    if (n == 0) return VX_OK;
    if (!world->trees_dev || !world_xyz_dev || !found_dev || !values_dev || !old_roots_dev || !edit_rank_dev ||
        world->chunk_depth < 0 || world->chunk_depth > 10)
        return VX_E_INVALID_ARG;
    uint64_t blocks = (n + 255) / 256;
    if (blocks > (uint64_t)num_sms * 16) blocks = (uint64_t)num_sms * 16;
    count_launches(1);
    if (D.vbits == 8)
        world_get_kernel<uint8_t><<<(unsigned)blocks, 256, 0, s>>>(D, *world, n, world_xyz_dev, found_dev,
                                                                   (uint8_t *)values_dev, old_roots_dev, edit_rank_dev,
                                                                   cut);
    else
        world_get_kernel<uint16_t><<<(unsigned)blocks, 256, 0, s>>>(D, *world, n, world_xyz_dev, found_dev,
                                                                    (uint16_t *)values_dev, old_roots_dev,
                                                                    edit_rank_dev, cut);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        interner_set_error(it, cudaGetErrorString(e));
        return VX_E_CUDA;
    }
    return VX_OK;
}

namespace vxg {
int interner_release_list(vx_interner *it, uint64_t *list_dev, int rounds);
}

extern "C" int vx_world_release_async(vx_interner *it, const vx_world *world, uint32_t n, const uint32_t *chunks_dev,
                                      uint64_t *held_dev, uint32_t *edit_rank_dev) {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false) || !world) return VX_E_INVALID_ARG;
    if (n == 0) return VX_OK;
    if (!world->trees_dev || !chunks_dev || !held_dev || !edit_rank_dev || world->chunk_depth < 0 ||
        world->chunk_depth > 10)
        return VX_E_INVALID_ARG;
    count_launches(1);
    world_unhold_kernel<<<(n + 255) / 256, 256, 0, s>>>(D, *world, n, chunks_dev, edit_rank_dev);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        interner_set_error(it, cudaGetErrorString(e));
        return VX_E_CUDA;
    }
    // dec_ref_recursive of every held root: a held root the apply replaced dies here
    return interner_release_list(it, held_dev, world->chunk_depth + 1);
}

// n host -> device copies on the interner's stream, one cudaMemcpyAsync each (serving loops stage a
// wave's arrays with one call instead of one runtime call per array from Python).
extern "C" int vx_copy_to_device_async(vx_interner *it, uint32_t n, void *const *dst_dev, const void *const *src_host,
                                       const uint64_t *bytes) {
    DevInterner D;
    cudaStream_t s;
    int num_sms;
    uint32_t flags;
    if (!interner_parts(it, &D, &s, &num_sms, &flags, false)) return VX_E_INVALID_ARG;
    if (n && (!dst_dev || !src_host || !bytes)) return VX_E_INVALID_ARG;
    for (uint32_t k = 0; k < n; ++k) {
        if (!bytes[k]) continue;
        const cudaError_t e = cudaMemcpyAsync(dst_dev[k], src_host[k], bytes[k], cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) {
            interner_set_error(it, cudaGetErrorString(e));
            return VX_E_CUDA;
        }
    }
    return VX_OK;
}
