// Path edits (src/device/pathedit.zig): voxels of a finished geometry are set,
// changed or removed without regenerating and rebuilding it. Only the path from
// the root to a changed brick is touched: the brick and the nodes above it are
// written as copies (new mask, voxel count and reference) into an arena above the
// geometry, everything else stays shared, so the node format and traversal are
// unchanged. Attributes are in depth-first order: an inserted or removed voxel
// shifts all later ones by one. RT prims point at subtrees: their node and the
// rank of their first voxel follow the change, and their boxes are recomputed.
//
// The reference runs one CTA per job and does everything of a job in it (thread 0
// walks, all threads then move the attributes). Here the parts are kernels over all
// jobs at once: the walks (one warp per job: a job's changes depend on each other
// through the root, but a node's words, its children's counts and the prims are read
// and written by the lanes together), the attribute map (one CTA per job), the attribute
// rewrite (over the whole GPU) and the boxes (one warp per prim). Every result equals the
// reference's job by job. 256 jobs of 32 edits over 200 M attributes: 0.58 ms a call, of
// which the attributes' 1.6 GB take 0.25 at the copy rate; 7.24 with a lane per walk and
// prim and with every attribute traced through all of its job's operations.
#pragma once

#include "pyrb_device.cuh"
#include "pyrb_internal.h"
#include "pyrb_kernels.cuh"

namespace pyrb {

// The reference's PathEditJob (src/device/types.zig:613-658), field for field.
struct PathEditJob {
    uint32_t node_offset, leaf_offset, root, log2_size;
    uint32_t attr_src, attr_count, attr_a, attr_b, attr_cap;
    uint32_t palette, pal_src, pal_dst;
    uint32_t node_arena, node_cap, leaf_arena, leaf_cap;
    uint32_t edit_first, edit_count, rt_log2, reserved0;
    uint64_t prims;
    uint32_t prim_count, reserved1;
    uint64_t aabbs;
    uint32_t aabbs_keep;
    uint32_t out_root, out_count, out_attr_b, out_flags;
    uint32_t op, op_rank, op_attr;
};
static_assert(sizeof(PathEditJob) == 136, "PathEditJob layout");

struct RtPrim {  // types.zig:518-525
    uint32_t node, attr_base;
    uint64_t cell;
};

constexpr uint32_t kPeOpNone = 0, kPeOpSet = 1, kPeOpInsert = 2, kPeOpRemove = 3;
constexpr uint32_t kPeRebuild = 0x1, kPeEmpty = 0x2, kPeOverflow = 0x4, kPeGrew = 0x8;
constexpr uint32_t kPeMaxEdits = 4096;   // types.path_edit_max_edits
constexpr uint32_t kPeStep = 4096;       // attributes per step of the rewrite
constexpr uint32_t kPeSteps = 4;
constexpr uint32_t kPeTile = kPeStep * kPeSteps;  // ... and per CTA
constexpr uint32_t kPePrimCache = 1024;  // prims of a job whose cells the walk keeps in shared memory
constexpr uint32_t kPeBoxWarps = kWarps;  // prims per CTA of the boxes

struct PathEditDesc {
    uint32_t* nodes;
    uint64_t* leaves;
    uint32_t* attrs;
    PathEditJob* jobs;
    const uint4* given;          // x, y, z, attribute, as the caller gave them
    uint4* edits;                // the same by brick (k_path_sort); the walk makes them (op, rank, value, 0), the
                                 // attribute map (what, place, value, 0)
    const uint32_t* attr_tile;   // [count + 1] first attribute tile of each job
    const uint32_t* prim_tile;   // [count + 1] first prim tile of each job
    uint32_t* places;            // [count] attributes of the job's target that come from its source or an operation
    uint32_t count;
};

__device__ __forceinline__ uint32_t pe_child_index(const uint32_t v[3], uint32_t s) {
    return ((v[0] >> s) & 1) | (((v[1] >> s) & 1) << 1) | (((v[2] >> s) & 1) << 2);
}
__device__ __forceinline__ uint64_t pe_morton(uint32_t x, uint32_t y, uint32_t z) {
    return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2);
}

struct PeWalker {
    uint32_t* nodes;
    uint64_t* leaves;
    uint32_t node_next, node_end, leaf_next, leaf_end;
    bool overflow;
    __device__ bool alloc_node(uint32_t words, uint32_t* out) {
        if (node_next + words > node_end) { overflow = true; return false; }
        *out = node_next;
        node_next += words;
        return true;
    }
    __device__ bool alloc_leaf(uint32_t* out) {
        if (leaf_next >= leaf_end) { overflow = true; return false; }
        *out = leaf_next++;
        return true;
    }
};

struct PeWalk {
    uint32_t missing;
    uint64_t brick;
    uint32_t prefix;
};

// Words of the nodes on the path to a brick, by level: [mask, count, references].
using PePath = uint32_t[kMaxLevels][kNodeStride];

// pathedit.zig:92-128: the path to the brick holding v and the rank of its first voxel.
// By the whole warp: a node's words in one load, the counts of the children before the
// path's one per lane and off the chain of dependent loads.
__device__ PeWalk pe_walk(const PeWalker& w, PePath& path, uint32_t root, uint32_t log2, const uint32_t v[3]) {
    const unsigned lane = threadIdx.x & 31;
    PeWalk r;
    r.missing = 0;
    r.brick = 0;
    uint32_t prefix = 0, node = root, s = log2 - 1;
    while (true) {
        // all words of a node at once where those behind a short node are still the pool's
        const bool whole = node + kNodeStride <= w.node_end;
        uint32_t word = lane < (whole ? kNodeStride : 2u) ? w.nodes[node + lane] : 0u;
        const uint32_t mask = __shfl_sync(kFull, word, 0) & 0xFF;
        if (!whole && lane >= 2 && lane < 2 + uint32_t(__popc(mask))) word = w.nodes[node + lane];
        if (lane < kNodeStride) path[s][lane] = word;
        const uint32_t ci = pe_child_index(v, s);
        const uint32_t before = __popc(mask & ((1u << ci) - 1));
        if (lane >= 2 && lane < 2 + before) prefix += s == 2 ? uint32_t(__popcll(w.leaves[word])) : w.nodes[word + 1];
        if (!(mask & (1u << ci))) { r.missing = s; break; }
        const uint32_t ref = __shfl_sync(kFull, word, 2 + before);
        if (s == 2) { r.brick = w.leaves[ref]; break; }
        node = ref;
        --s;
    }
    r.prefix = __reduce_add_sync(kFull, prefix);
    __syncwarp();  // the path's words
    return r;
}

// pathedit.zig:137-193: copies of the path with the new brick; false on arena overflow.
// By the whole warp, lane k writing word k of a node.
__device__ bool pe_rewrite(PeWalker& w, const PePath& path, const PeWalk& wk, uint32_t log2, uint32_t sub_level,
                           const uint32_t v[3], uint64_t new_brick, int32_t delta, bool* has_root, uint32_t* root,
                           bool* has_sub, uint32_t* sub) {
    const unsigned lane = threadIdx.x & 31;
    bool has_child = false;
    uint32_t child = 0;
    if (new_brick != 0) {
        uint32_t l;
        if (!w.alloc_leaf(&l)) return false;
        if (lane == 0) w.leaves[l] = new_brick;
        child = l;
        has_child = true;
    }
    *has_sub = false;
    for (uint32_t s = 2; s < log2; ++s) {
        const uint32_t ci = pe_child_index(v, s), cbit = 1u << ci;
        const bool exists = wk.missing == 0 || s >= wk.missing;
        const uint32_t om = exists ? path[s][0] & 0xFF : 0u;
        const uint32_t mask = has_child ? om | cbit : om & ~cbit;
        const uint32_t count = (exists ? path[s][1] : 0u) + uint32_t(delta);
        if (mask == 0) {
            has_child = false;
        } else {
            const uint32_t n = __popc(mask);
            uint32_t nn;
            if (!w.alloc_node(2 + n, &nn)) return false;
            uint32_t word = lane == 0 ? mask : count;
            if (lane >= 2 && lane < 2 + n) {
                const uint32_t k = __fns(mask, 0, int(lane) - 1);  // the child of reference lane - 2
                word = k == ci ? child : path[s][2 + __popc(om & ((1u << k) - 1))];
            }
            if (lane < 2 + n) w.nodes[nn + lane] = word;
            child = nn;
            has_child = true;
        }
        if (s + 1 == sub_level) { *has_sub = has_child; *sub = child; }
    }
    *has_root = has_child;
    *root = child;
    __syncwarp();  // the next walk reads what other lanes wrote
    return true;
}

// A job's prims during its walk: their cells' Morton codes and the changes of their
// attribute ranks, the first kPePrimCache of them in shared memory.
struct PePrims {
    uint64_t cell[kPePrimCache];
    uint32_t shift[kPePrimCache];
};
__device__ __forceinline__ uint64_t pe_prim_cell(const RtPrim* prims, uint32_t k) {
    const uint64_t c = prims[k].cell;
    return pe_morton(uint32_t(c & 0x1FFFFF), uint32_t((c >> 21) & 0x1FFFFF), uint32_t((c >> 42) & 0x1FFFFF));
}

// pathedit.zig:489-534: prims follow the change of the brick at v
__device__ void pe_update_prims(PeWalker& w, PePrims& cache, const PathEditJob& job, const uint32_t v[3], int32_t delta,
                                bool has_sub, uint32_t sub, uint32_t* flags) {
    if (!job.prims) return;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t mc = pe_morton(v[0] >> job.rt_log2, v[1] >> job.rt_log2, v[2] >> job.rt_log2);
    RtPrim* prims = reinterpret_cast<RtPrim*>(job.prims);
    const uint32_t n = job.prim_count;
    bool found = false;
    for (uint32_t k0 = 0; k0 < n; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool in = k < n;
        const uint64_t mp = !in ? 0 : k < kPePrimCache ? cache.cell[k] : pe_prim_cell(prims, k);
        const unsigned hits = __ballot_sync(kFull, in && mp == mc);
        if (hits) {
            found = true;
            if (has_sub) {
                if ((hits >> lane) & 1) prims[k].node = sub;
            } else {
                for (unsigned h = hits; h; h &= h - 1) {  // in prim order: each takes an empty node
                    uint32_t en;
                    if (!w.alloc_node(2, &en)) {
                        *flags |= kPeOverflow;
                    } else if (lane == uint32_t(__ffs(h)) - 1) {
                        w.nodes[en] = 0;
                        w.nodes[en + 1] = 0;
                        prims[k].node = en;
                    }
                }
            }
        }
        if (in && mp > mc) {
            if (k < kPePrimCache) cache.shift[k] += uint32_t(delta);
            else prims[k].attr_base += uint32_t(delta);
        }
    }
    if (!found && has_sub) *flags |= kPeRebuild;
}

__device__ __forceinline__ PeWalker pe_walker(const PathEditDesc& p, const PathEditJob& job) {
    PeWalker w;
    w.nodes = p.nodes + job.node_offset;
    w.leaves = p.leaves + job.leaf_offset;
    w.node_next = job.node_arena - job.node_offset;
    w.node_end = job.node_arena - job.node_offset + job.node_cap;
    w.leaf_next = job.leaf_arena - job.leaf_offset;
    w.leaf_end = job.leaf_arena - job.leaf_offset + job.leaf_cap;
    w.overflow = false;
    return w;
}

// 0. Each job's edits stably ordered by brick, so that a brick is one run and gets one new
// path (Context.pathEdit's sort on the host). One CTA per job: an edit's place is the
// number of edits before it, counted over the keys in shared memory (32 edits take a few
// us, the 4096 a job may have 0.2 ms; 256 sorts of 32 took the host 0.15 ms).
__global__ void __launch_bounds__(kBlock) k_path_sort(PathEditDesc p) {
    grid_dep_wait();
    extern __shared__ uint64_t s_brick[];  // [largest edit_count of the jobs]
    const PathEditJob& job = p.jobs[blockIdx.x];
    const uint32_t n = min(job.edit_count, kPeMaxEdits);
    const uint4* in = p.given + job.edit_first;
    uint4* out = p.edits + job.edit_first;
    for (uint32_t k = threadIdx.x; k < n; k += kBlock) {
        const uint4 e = in[k];
        s_brick[k] = uint64_t(e.z >> 2) << 42 | uint64_t(e.y >> 2) << 21 | uint64_t(e.x >> 2);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n; k += kBlock) {
        const uint64_t me = s_brick[k];
        uint32_t place = 0;
        for (uint32_t q = 0; q < n; ++q) place += s_brick[q] < me || (s_brick[q] == me && q < k) ? 1u : 0u;
        out[place] = in[k];
    }
}

// 1. One warp per job walks the job's bricks in order (pathedit.zig:283-368).
__global__ void __launch_bounds__(32) k_path_walk(PathEditDesc p) {
    grid_dep_wait();
    __shared__ PePath s_path;
    __shared__ PePrims s_prims;
    __shared__ uint32_t s_pal[16];
    const uint32_t j = blockIdx.x;
    const unsigned lane = threadIdx.x;
    PathEditJob& out = p.jobs[j];
    const PathEditJob job = out;
    PeWalker w = pe_walker(p, job);
    uint4* edits = p.edits + job.edit_first;
    const uint32_t n_edits = job.edit_count;
    uint32_t n_pal = 0;
    if (job.palette) {
        if (lane < 16) s_pal[lane] = p.attrs[job.pal_src + lane];
        __syncwarp();
        // entries up to the first repeat of entry 0 (the padding)
        const unsigned rep = __ballot_sync(kFull, lane >= 1 && lane < 16 && s_pal[lane] == s_pal[0]);
        n_pal = rep ? uint32_t(__ffs(rep)) - 1 : 16u;
    }
    RtPrim* prims = reinterpret_cast<RtPrim*>(job.prims);
    const uint32_t cached = prims ? min(job.prim_count, kPePrimCache) : 0u;
    for (uint32_t k = lane; k < cached; k += 32) {
        s_prims.cell[k] = pe_prim_cell(prims, k);
        s_prims.shift[k] = 0;
    }
    __syncwarp();
    uint32_t root = job.root, flags = 0, count = job.attr_count;
    int32_t undone = 0;  // voxels that a brick gained whose path found no room
    uint32_t e = 0;
    while (e < n_edits) {
        const uint4 lead = edits[e];
        const uint32_t v0[3] = {lead.x, lead.y, lead.z};
        // the edits of the brick: a stretch of the sorted list, 32 looked at together
        uint32_t end = e + 1;
        for (bool more = true; more;) {
            const uint32_t k = end + lane;
            bool same = false;
            if (k < n_edits) {
                const uint4 q = edits[k];
                same = (q.x >> 2) == (v0[0] >> 2) && (q.y >> 2) == (v0[1] >> 2) && (q.z >> 2) == (v0[2] >> 2);
            }
            const unsigned other = __ballot_sync(kFull, !same);
            end += other ? uint32_t(__ffs(other)) - 1 : 32u;
            more = other == 0;
        }
        if (flags & (kPeEmpty | kPeOverflow)) {
            for (uint32_t k = e + lane; k < end; k += 32) edits[k] = make_uint4(kPeOpNone, 0, edits[k].w, 0);
            e = end;
            __syncwarp();
            continue;
        }
        const PeWalk wk = pe_walk(w, s_path, root, job.log2_size, v0);
        uint64_t brick = wk.brick;
        int32_t delta = 0;
        for (; e < end; ++e) {
            const uint4 q = edits[e];
            __syncwarp();  // read by every lane before lane 0 overwrites it
            const uint32_t bit = (q.x & 3) + 4 * (q.y & 3) + 16 * (q.z & 3);
            const uint64_t bm = uint64_t(1) << bit;
            const uint32_t rank = wk.prefix + uint32_t(__popcll(brick & (bm - 1)));
            const bool has = (brick & bm) != 0;
            uint32_t val = q.w;
            if (job.palette && q.w != 0) {
                const unsigned hit = __ballot_sync(kFull, lane < n_pal && s_pal[lane & 15] == val);
                uint32_t idx = hit ? uint32_t(__ffs(hit)) - 1 : n_pal;
                if (!hit) {
                    if (n_pal == 16) {
                        flags |= kPeOverflow;
                        if (lane == 0) edits[e] = make_uint4(0, 0, 0, 0);
                        continue;
                    }
                    if (lane == 0) s_pal[n_pal] = val;
                    ++n_pal;
                    __syncwarp();
                }
                val = idx;
            }
            uint32_t op = kPeOpNone;
            if (q.w != 0 && has) op = kPeOpSet;
            if (q.w != 0 && !has) { op = kPeOpInsert; brick |= bm; delta += 1; }
            if (q.w == 0 && has) { op = kPeOpRemove; brick &= ~bm; delta -= 1; }
            if (lane == 0) edits[e] = make_uint4(op, rank, val, 0);
        }
        if (brick != wk.brick) {
            bool has_root, has_sub;
            uint32_t nr = 0, sub = 0;
            if (!pe_rewrite(w, s_path, wk, job.log2_size, job.rt_log2, v0, brick, delta, &has_root, &nr, &has_sub, &sub)) {
                flags |= kPeOverflow;
                undone = delta;
                continue;
            }
            if (has_root) root = nr; else flags |= kPeEmpty;
            count = uint32_t(int32_t(count) + delta);
            pe_update_prims(w, s_prims, job, v0, delta, has_sub, sub, &flags);
        }
    }
    if (w.overflow) flags |= kPeOverflow;
    __syncwarp();
    for (uint32_t k = lane; k < cached; k += 32)
        if (s_prims.shift[k]) prims[k].attr_base += s_prims.shift[k];
    if (job.palette && lane < 16) p.attrs[job.pal_dst + lane] = lane < n_pal ? s_pal[lane] : s_pal[0];
    if (lane == 0) {
        out.out_root = root;
        out.out_count = count;
        out.out_attr_b = 0;
        out.out_flags = flags;
        // The operations of a brick whose path found no room stay in the list, but the tree
        // and the count are those before it. With more removals than inserts among them the
        // list is shorter than the count: the places behind it have no source (they would come
        // from behind the job's attributes), and the map makes them 0. (The result of such a
        // job is not used.)
        p.places[j] = flags & kPeEmpty ? 0u : undone < 0 ? count - uint32_t(-undone) : count;
    }
}

// 2. The attributes after all operations come from those before them (pathedit.zig:
// 462-485 traces every attribute back through all of the job's operations; here every
// operation is traced once, so that an attribute only meets those near it). In place of
// an operation:
//   kPeMapInsert  the attribute at `place` is `value`, and those after it come one later
//   kPeMapSet     the attribute at `place` is `value`
//   kPeMapRemove  the attributes from `place` on come one earlier
//   0             none of these: overtaken by a later removal, or the removal of a voxel
//                 that the job inserted
// An attribute i whose place no operation took has the old rank
//   i - #{inserts at places < i} + #{removals at places <= i};
// of several operations that took a place the last one counts. One CTA per job, the
// operations staged in shared memory.
constexpr uint32_t kPeMapInsert = 1, kPeMapSet = 2, kPeMapRemove = 3;
__global__ void __launch_bounds__(kBlock) k_path_map(PathEditDesc p) {
    grid_dep_wait();
    extern __shared__ uint2 s_op[];  // [largest edit_count of the jobs]: op, rank
    const PathEditJob& job = p.jobs[blockIdx.x];
    const uint32_t n = min(job.edit_count, kPeMaxEdits);
    uint4* ops = p.edits + job.edit_first;
    for (uint32_t k = threadIdx.x; k < n; k += kBlock) s_op[k] = make_uint2(ops[k].x, ops[k].y);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n; k += kBlock) {
        const uint2 o = s_op[k];
        uint32_t what = 0, place = o.y;
        if (o.x == kPeOpRemove) {
            what = kPeMapRemove;
            uint32_t idx = o.y;  // back: is it a voxel that the job inserted?
            for (uint32_t q = k; q > 0;) {
                const uint2 b = s_op[--q];
                if (b.x == kPeOpInsert) {
                    if (idx == b.y) { what = 0; break; }
                    if (idx > b.y) --idx;
                } else if (b.x == kPeOpRemove) {
                    if (idx >= b.y) ++idx;
                }
            }
            // forward: the place between two attributes
            for (uint32_t q = k + 1; q < n; ++q) {
                const uint2 b = s_op[q];
                if (b.x == kPeOpInsert) place += place > b.y ? 1u : 0u;
                else if (b.x == kPeOpRemove) place -= place > b.y ? 1u : 0u;
            }
        } else if (o.x != kPeOpNone) {
            what = o.x == kPeOpInsert ? kPeMapInsert : kPeMapSet;
            for (uint32_t q = k + 1; q < n; ++q) {
                const uint2 b = s_op[q];
                if (b.x == kPeOpInsert) {
                    place += place >= b.y ? 1u : 0u;
                } else if (b.x == kPeOpRemove) {
                    if (place == b.y) { what = 0; break; }
                    place -= place > b.y ? 1u : 0u;
                }
            }
        }
        ops[k].x = what;
        ops[k].y = place;
    }
    if (job.out_flags & kPeEmpty) return;
    // (the word of the last place that has a source is the rewrite's)
    const uint32_t per = job.palette ? 8 : 1, end = (job.out_count + per - 1) / per;
    uint32_t* dst = p.attrs + job.attr_a;
    for (uint32_t i = (p.places[blockIdx.x] + per - 1) / per + threadIdx.x; i < end; i += kBlock) dst[i] = 0;
}

// 3. Attributes of every job, kPeTile outputs per CTA in kPeSteps steps (pathedit.zig:
// 370-425). The CTA adds up the operations before each of its steps; a step that none of
// them lies in is a copy at one distance, else the distances come from a scan over the
// step in shared memory. Four steps per CTA share its look-ups, which are five round trips
// before the first copy: 200 M attributes take 354 us, 656 with one step (316 since the ends
// of a step are differences).
__global__ void __launch_bounds__(kBlock) k_path_attrs(PathEditDesc p) {
    grid_dep_wait();
    __shared__ int32_t s_dist[kPeStep];   // old rank - new rank
    __shared__ uint32_t s_took[kPeStep];  // the last operation (+ 1) that took the place
    __shared__ uint32_t s_scan[2 * kWarps + 2];
    __shared__ uint32_t s_before[kWarps][kPeSteps + 1];  // per step; whether an operation lies in it
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x;
    const uint32_t j = warp_upper_index(p.attr_tile, p.count + 1, tile);
    if (j >= p.count) return;
    const PathEditJob& job = p.jobs[j];
    const uint32_t n_ops = min(job.edit_count, kPeMaxEdits), n_final = p.places[j];
    const uint32_t tile0 = (tile - __ldg(p.attr_tile + j)) * kPeTile;
    if (tile0 >= n_final) return;
    const uint4* ops = p.edits + job.edit_first;
    {
        uint32_t before[kPeSteps] = {}, inside = 0;  // (differences: may wrap)
        for (uint32_t k = threadIdx.x; k < n_ops; k += kBlock) {
            const uint4 o = ops[k];
            if (o.x == 0) continue;
#pragma unroll
            for (uint32_t s = 0; s < kPeSteps; ++s) {
                const uint32_t t0 = tile0 + s * kPeStep;
                if (o.x == kPeMapInsert) before[s] -= o.y < t0 ? 1u : 0u;
                if (o.x == kPeMapRemove) before[s] += o.y <= t0 ? 1u : 0u;
                if (o.y - t0 < kPeStep) inside |= 1u << s;
            }
        }
#pragma unroll
        for (uint32_t s = 0; s < kPeSteps; ++s) {
            const uint32_t sum = __reduce_add_sync(kFull, before[s]);
            if (lane == 0) s_before[warp][s] = sum;
        }
        inside = __reduce_or_sync(kFull, inside);
        if (lane == 0) s_before[warp][kPeSteps] = inside;
    }
    __syncthreads();
    uint32_t in_steps = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) in_steps |= s_before[w][kPeSteps];
    constexpr uint32_t kPer = kPeStep / kBlock;
    const uint32_t* src = p.attrs + job.attr_src;
    uint32_t* dst = p.attrs + job.attr_a;
    for (uint32_t s = 0; s < kPeSteps; ++s) {
        if (n_final - tile0 <= s * kPeStep) break;  // (differences: a step's end may lie beyond 32 bits)
        const uint32_t t0 = tile0 + s * kPeStep, m = min(n_final - t0, kPeStep);
        const bool inside = (in_steps >> s) & 1;
        uint32_t dist0 = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) dist0 += s_before[w][s];
        if (inside) {
            __syncthreads();  // the step before is done with the arrays
            for (uint32_t k = threadIdx.x; k < kPeStep; k += kBlock) { s_dist[k] = 0; s_took[k] = 0; }
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < n_ops; k += kBlock) {
                const uint4 o = ops[k];
                if (o.x == 0 || o.y - t0 >= kPeStep) continue;
                const uint32_t i = o.y - t0;
                if (o.x == kPeMapRemove) {
                    if (i > 0) atomicAdd(s_dist + i, 1);
                } else {
                    atomicMax(s_took + i, k + 1);
                    if (o.x == kPeMapInsert && i + 1 < kPeStep) atomicAdd(s_dist + i + 1, -1);
                }
            }
            __syncthreads();
            uint32_t sum = 0, unused;
#pragma unroll
            for (uint32_t k = 0; k < kPer; ++k) sum += uint32_t(s_dist[threadIdx.x * kPer + k]);
            uint32_t run = dist0 + block_excl_scan(sum, s_scan, &unused);
#pragma unroll
            for (uint32_t k = 0; k < kPer; ++k) {
                run += uint32_t(s_dist[threadIdx.x * kPer + k]);
                s_dist[threadIdx.x * kPer + k] = int32_t(run);
            }
            __syncthreads();
        }
        if (job.palette) {
            for (uint32_t wd = t0 / 8 + threadIdx.x; wd < t0 / 8 + (m + 7) / 8; wd += kBlock) {
                const uint32_t i0 = wd * 8, n = min(n_final - i0, 8u);
                uint32_t word = 0;
                if (!inside) {
                    const uint32_t a = i0 + dist0, b = a + n - 1;
                    const uint32_t lo = src[a >> 3], hi = (b >> 3) != (a >> 3) ? src[b >> 3] : 0u;
                    word = __funnelshift_r(lo, hi, (a & 7) * 4);
                    if (n < 8) word &= (1u << (4 * n)) - 1;
                } else {
                    for (uint32_t q = 0; q < n; ++q) {
                        const uint32_t i = i0 + q - t0, took = s_took[i];
                        const uint32_t idx = t0 + i + uint32_t(s_dist[i]);
                        const uint32_t x = took ? ops[took - 1].z : (src[idx >> 3] >> ((idx & 7) * 4)) & 15;
                        word |= x << (q * 4);
                    }
                }
                dst[wd] = word;
            }
            continue;
        }
        // (a job's target never overlaps its source)
        uint32_t v[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t i = threadIdx.x + k * kBlock;
            v[k] = 0;
            if (i >= m) continue;
            const uint32_t took = inside ? s_took[i] : 0u;
            v[k] = took ? ops[took - 1].z : src[t0 + i + (inside ? uint32_t(s_dist[i]) : dist0)];
        }
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k)
            if (threadIdx.x + k * kBlock < m) dst[t0 + threadIdx.x + k * kBlock] = v[k];
    }
}

// pathedit.zig:198-236: tight box of a subtree in its own coordinates
__device__ void pe_subtree_box(const PeWalker& w, uint32_t node, uint32_t s_top, uint32_t lo[3], uint32_t hi[3]) {
    for (int a = 0; a < 3; ++a) { lo[a] = 0xFFFFFFFFu; hi[a] = 0; }
    struct Entry { uint32_t node, s, off[3]; };
    Entry stack[64];
    uint32_t sp = 1;
    stack[0] = {node, s_top, {0, 0, 0}};
    while (sp > 0) {
        const Entry e = stack[--sp];
        const uint32_t mask = w.nodes[e.node] & 0xFF, size = 1u << e.s;
        uint32_t slot = 0;
        for (uint32_t k = 0; k < 8; ++k) {
            if (!(mask & (1u << k))) continue;
            const uint32_t ref = w.nodes[e.node + 2 + slot];
            ++slot;
            const uint32_t off[3] = {e.off[0] + (k & 1) * size, e.off[1] + ((k >> 1) & 1) * size,
                                     e.off[2] + (k >> 2) * size};
            if (e.s == 2) {
                const uint64_t brick = w.leaves[ref];
                for (uint32_t b = 0; b < 64; ++b) {
                    if (!((brick >> b) & 1)) continue;
                    const uint32_t v[3] = {off[0] + (b & 3), off[1] + ((b >> 2) & 3), off[2] + (b >> 4)};
                    for (int a = 0; a < 3; ++a) {
                        lo[a] = min(lo[a], v[a]);
                        hi[a] = max(hi[a], v[a] + 1);
                    }
                }
            } else if (sp < 64) {
                stack[sp++] = {ref, e.s - 1, {off[0], off[1], off[2]}};
            }
        }
    }
}

// The same by a whole warp for subtrees up to 2^kPeBoxLog2: four nodes at a time, a lane
// per child; subtrees inside the box found so far are passed over.
constexpr uint32_t kPeBoxLog2 = 10;
constexpr uint32_t kPeBoxStack = 28 * (kPeBoxLog2 - 2) + 40;  // 4 leave, up to 32 come, once per level
struct PeBoxNode { uint32_t node, level, x, y, z; };
__device__ void pe_subtree_box_warp(const PeWalker& w, PeBoxNode* stack, uint32_t node, uint32_t s_top, uint32_t lo[3],
                                    uint32_t hi[3]) {
    const unsigned lane = threadIdx.x & 31;
    for (int a = 0; a < 3; ++a) { lo[a] = 0xFFFFFFFFu; hi[a] = 0; }
    uint32_t sp = 1;
    if (lane == 0) stack[0] = {node, s_top, 0, 0, 0};
    __syncwarp();
    while (sp > 0) {
        const uint32_t take = min(sp, 4u), g = lane >> 3, k = lane & 7;
        bool push = false;
        PeBoxNode c = {};
        if (g < take) {
            const PeBoxNode e = stack[sp - 1 - g];
            const uint32_t edge = 2u << e.level;  // the node's own
            const bool inside = lo[0] <= e.x && lo[1] <= e.y && lo[2] <= e.z && hi[0] >= e.x + edge &&
                                hi[1] >= e.y + edge && hi[2] >= e.z + edge;
            if (!inside) {
                const uint32_t mask = w.nodes[e.node] & 0xFF, size = 1u << e.level;
                if (mask & (1u << k)) {
                    const uint32_t ref = w.nodes[e.node + 2 + __popc(mask & ((1u << k) - 1))];
                    c = {ref, e.level - 1, e.x + (k & 1) * size, e.y + ((k >> 1) & 1) * size, e.z + (k >> 2) * size};
                    if (e.level == 2) {
                        const uint64_t brick = w.leaves[ref];
                        if (brick) {
                            uint64_t blo, bhi;
                            brick_box(brick, blo, bhi);
                            lo[0] = min(lo[0], c.x + cell_x(blo)); hi[0] = max(hi[0], c.x + cell_x(bhi));
                            lo[1] = min(lo[1], c.y + cell_y(blo)); hi[1] = max(hi[1], c.y + cell_y(bhi));
                            lo[2] = min(lo[2], c.z + cell_z(blo)); hi[2] = max(hi[2], c.z + cell_z(bhi));
                        }
                    } else {
                        push = true;
                    }
                }
            }
        }
        sp -= take;
        __syncwarp();
        const unsigned pushed = __ballot_sync(kFull, push);
        // the top node's children end on top: the stack stays ordered by level, at most 28
        // nodes of each but the first
        if (push) stack[sp + __popc(pushed >> lane >> 1)] = c;
        sp += __popc(pushed);
        for (int a = 0; a < 3; ++a) {
            lo[a] = __reduce_min_sync(kFull, lo[a]);
            hi[a] = __reduce_max_sync(kFull, hi[a]);
        }
        __syncwarp();
    }
}

// 4. Boxes of every prim of every job (pathedit.zig:427-459), one warp per prim.
__global__ void __launch_bounds__(kBlock) k_path_boxes(PathEditDesc p) {
    grid_dep_wait();
    __shared__ PeBoxNode s_stack[kPeBoxWarps][kPeBoxStack];
    const uint32_t tile = blockIdx.x;
    const uint32_t j = warp_upper_index(p.prim_tile, p.count + 1, tile);
    if (j >= p.count) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PathEditJob& job = p.jobs[j];
    const uint32_t k = (tile - __ldg(p.prim_tile + j)) * kPeBoxWarps + warp;
    if (!job.aabbs || !job.prims || k >= job.prim_count) return;
    const PeWalker w = pe_walker(p, job);
    const RtPrim* prims = reinterpret_cast<const RtPrim*>(job.prims);
    float* box_out = reinterpret_cast<float*>(job.aabbs) + uint64_t(k) * 6;
    const uint32_t size = 1u << job.rt_log2;
    const float eps = 1.0f / 256.0f;
    const uint64_t c = prims[k].cell;
    const uint32_t cell[3] = {uint32_t(c & 0x1FFFFF), uint32_t((c >> 21) & 0x1FFFFF), uint32_t((c >> 42) & 0x1FFFFF)};
    uint32_t lo[3], hi[3];
    // larger subtrees take the reference's depth-first order with its stack of 64
    if (job.rt_log2 <= kPeBoxLog2) pe_subtree_box_warp(w, s_stack[warp], prims[k].node, job.rt_log2 - 1, lo, hi);
    else if (lane == 0) pe_subtree_box(w, prims[k].node, job.rt_log2 - 1, lo, hi);
    if (lane != 0) return;
    if (lo[0] > hi[0]) { lo[0] = lo[1] = lo[2] = 0; hi[0] = hi[1] = hi[2] = 0; }
    float box[6];
    for (int a = 0; a < 3; ++a) {
        const float base = float(cell[a] * size);
        box[a] = __fsub_rn(__fadd_rn(base, float(lo[a])), eps);
        box[3 + a] = __fadd_rn(__fadd_rn(base, float(hi[a])), eps);
    }
    bool grew = false;
    if (!job.aabbs_keep) {
        for (int a = 0; a < 6; ++a) box_out[a] = box[a];
        grew = true;
    } else {
        bool inside = true;
        for (int a = 0; a < 3; ++a)
            if (box[a] < box_out[a] || box[3 + a] > box_out[3 + a]) inside = false;
        if (!inside) {
            for (int a = 0; a < 3; ++a) {
                const float base = float(cell[a] * size);
                box_out[a] = __fsub_rn(base, eps);
                box_out[3 + a] = __fadd_rn(__fadd_rn(base, float(size)), eps);
            }
            grew = true;
        }
    }
    if (grew) atomicOr(&job.out_flags, kPeGrew);
}

}  // namespace pyrb
