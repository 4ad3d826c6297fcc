// gpu_bvh.cu -- the reference's binned-SAH AABB tree (src/aabbTreeBuilder.cpp:
// 52-214) built on the GPU, byte-identical to host_build_bvh.
//
// The reference builds breadth-first from a FIFO queue and numbers nodes in
// pop order, so a node's number is its rank by (level, first leaf position).
// A range of leaves is split without knowing that number, so the build has
// three phases:
//   1. ranges of more than kSmall leaves ("big"), one tree level per round of
//      kernels over chunks of kChunk leaves of one range each:
//        bucket   12 centroid buckets per range, per block in shared memory;
//        sah      one warp per range: the reference's split sweep with the
//                 same float operations; the left leaves before each chunk;
//        next     the next level's ranges in position order;
//        part     every leaf's rank among its side (the stable partition);
//        move     leaves to their places, and the bounds of both halves.
//      The host waits once for all levels (the kernels read the range count
//      from device memory and are empty when none is left).
//   2. every range of 2 to kSmall leaves: one warp builds its whole subtree
//      from shared memory, breadth first.
//   3. numbering: nodes per (level, subtree), a scan of each level over the
//      subtrees in position order, and the records written with final links.
// The partition is the reference's in-place loop
//   for i: if bucket[i] <= opt: swap(a[i], a[pivot++])
// The right-hand leaves between pivot and i behave as a queue: a left leaf at
// i moves the queue's front to i, a right leaf appends itself.  So the leaf
// that ends at place q >= beg + nL is found backwards: p = q; while the leaf
// at p is a left one, p = beg + (left leaves before p).  Over a run of left
// leaves that step is a subtraction of the constant r = right leaves before
// p, so a whole run is crossed at once.
// Min and max are order-independent (no NaN; -0 made +0 as the reference's
// world-matrix multiply does), so reductions may run in any order.
//
// What bounds it: phase 1 moves about 110 bytes per leaf and level, from L2
// (a level of 1.05M leaves takes 65 us: move 26, bucket 16, sah 9, part 8,
// next 8); phase 2 is bound by instruction issue, about 500 a node.  Measured
// at 1.05M triangles: 1.72 ms, against 13.1 ms for a round of 45 launches over
// all leaves at every one of the 26 levels with 18 allocations a call; at
// 20,012 triangles 0.6 ms, at 780 0.3 ms (5 ms before).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include <string.h>

#include "rg_internal.h"

namespace {

constexpr int kBuckets = 12;
#ifndef RG_BVH_SMALL
#define RG_BVH_SMALL 128
#endif
// Leaves of a range that one warp takes whole: 1.05M triangles build in 2.13,
// 1.84, 1.72 ms with 32, 64, 128 (a level of phase 1 costs more than the
// warps' longer chains); 128 is the most that places in bytes allow.
constexpr int kSmall = RG_BVH_SMALL;
constexpr int kChunk = 1024;          // leaves of a block's share of a big range
constexpr int kBlock = 256;

// A leaf: its box (the centroid is 0.5 * (lo + hi), recomputed where needed).
struct Leaf {
    float4 a;  // lo.xyz, triangle (int bits)
    float4 b;  // hi.xyz, 0
};
__device__ __forceinline__ float3 centroid(const Leaf &l) {
    return make_float3(0.5f * (l.a.x + l.b.x), 0.5f * (l.a.y + l.b.y), 0.5f * (l.a.z + l.b.z));
}
__device__ __forceinline__ float axis_of(float3 v, int d) { return d == 0 ? v.x : d == 1 ? v.y : v.z; }

// float -> int key with the same order (no NaN); involution on negatives
__host__ __device__ __forceinline__ int fkey(float f) {
    int b;
    memcpy(&b, &f, 4);
    return b >= 0 ? b : b ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float kfloat(int k) {
    const int b = k >= 0 ? k : k ^ 0x7fffffff;
    float f;
    memcpy(&f, &b, 4);
    return f;
}
// keys of FLT_MAX and -FLT_MAX: the empty box
constexpr int kKeyMax = 0x7f7fffff, kKeyMin = (int)0x80800000;
// nvmath nv_min / nv_max
__device__ __forceinline__ float nvmin(float a, float b) { return (a < b) ? a : b; }
__device__ __forceinline__ float nvmax(float a, float b) { return (a > b) ? a : b; }

__device__ __forceinline__ float surface_area(const float *mn, const float *mx) {
    const float sx = mx[0] - mn[0], sy = mx[1] - mn[1], sz = mx[2] - mn[2];
    return (sx * sy + sx * sz) + sy * sz;
}

// A big range of one level.  Keys: [0..2] centroid min, [3..5] centroid max,
// [6..8] box min, [9..11] box max; buckets: 3 min and 3 max keys of the boxes.
struct Task {
    int32_t keys[12];
    int32_t bcount[kBuckets];
    int32_t bkeys[kBuckets][6];
    int32_t opt, nl, fallback;
    int32_t hkeys[12];            // median split: box min, max keys of the left then the right half
};
// Its place, in an array of its own for the single-block kernel that makes
// the next level: (beg, end, first chunk, chunks), and after the split
// (pivot, index of a big left half in the next level or -1, right half).
struct Range {
    int32_t beg, end, chunk0, chunks;
};
struct Split {
    int32_t pivot, child[2], pad;
};
struct Chunk {
    int32_t task, beg, end;
    int32_t left;                 // left leaves of the range before this chunk
};

// A node before numbering, 64 bytes.  A node is stored at the gap it belongs
// to: a big range at slot pivot - 1, node i of a subtree at slot beg + i (its
// ranges' gaps are beg .. end - 2), so every slot is used once.
struct Rec {
    float box[12];                // left min, left max, right min, right max
    int32_t l, r;                 // big: beg, end; subtree: ~triangle or the child's rank among the
                                  // subtree's nodes of the next level
    int32_t level, rank;          // big: level, index among the level's big ranges; subtree: level and rank
                                  // within the subtree
};
struct Subtree {
    int32_t beg, end, level;
};

struct Ctrl {
    int32_t tasks[2], chunks[2];  // of the level with that parity
    int32_t bigs;                 // big ranges of all levels so far
    int32_t max_level;            // deepest level of any node
    int32_t undefined;
    int32_t subtrees;
};

// The empty statistics of a range, by the lanes of one warp.
__device__ __forceinline__ void clear_task(Task &t, int lane) {
    for (int j = lane; j < 12; j += 32) {
        t.keys[j] = (j % 6) < 3 ? kKeyMax : kKeyMin;
        t.hkeys[j] = (j % 6) < 3 ? kKeyMax : kKeyMin;
        t.bcount[j] = 0;
    }
    for (int j = lane; j < kBuckets * 6; j += 32) t.bkeys[j / 6][j % 6] = (j % 6) < 3 ? kKeyMax : kKeyMin;
}

__device__ __forceinline__ int bucket_of(float c, float cmin, float range, int undefined) {
    float u = undefined ? 0.5f : (c - cmin) / range;
    u = (u < 0.5f) ? 0.5f : u;
    u = (u > (float)kBuckets - 0.5f) ? (float)kBuckets - 0.5f : u;
    return (int)u;
}

// The widest centroid axis, as the reference picks it; outer = area of the box.
struct Axis {
    int dim, undefined;
    float cmin, range, outer;
};
__device__ __forceinline__ Axis pick_axis(const int *k) {
    float cmin[3], cmax[3], amin[3], amax[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        cmin[d] = kfloat(k[d]);
        cmax[d] = kfloat(k[3 + d]);
        amin[d] = kfloat(k[6 + d]);
        amax[d] = kfloat(k[9 + d]);
    }
    Axis a;
    a.outer = surface_area(amin, amax);
    const float sx = cmax[0] - cmin[0], sy = cmax[1] - cmin[1], sz = cmax[2] - cmin[2];
    a.dim = sx > sy ? 0 : 1;
    float span = sx > sy ? sx : sy;
    a.cmin = sx > sy ? cmin[0] : cmin[1];
    if (sz > span) {
        a.dim = 2;
        span = sz;
        a.cmin = cmin[2];
    }
    a.range = span / (float)kBuckets;
    a.undefined = (!(a.range > 0.0f) || !(a.outer > 0.0f)) ? 1 : 0;
    return a;
}

// The reference's split sweep (aabbTreeBuilder.cpp:146-173) by one warp: lane
// b < 12 holds bucket b's count and box; lane s < 11 evaluates the split after
// bucket s from a prefix and a suffix merge over the lanes.  The first split
// with the strictly smallest heuristic wins; a NaN heuristic (an empty side)
// never does.  Returns the winning lane or -1; lb, rb are this lane's boxes
// (min then max), lc this lane's left count.
__device__ __forceinline__ int sah_warp(int lane, int cnt, const int *key6, float outer, float *lb, float *rb,
                                        int &lc) {
    constexpr unsigned kFull = 0xffffffffu;
    int l[6], r[6], rc = cnt;
    lc = cnt;
#pragma unroll
    for (int d = 0; d < 6; ++d) l[d] = r[d] = key6[d];
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int lcn = __shfl_up_sync(kFull, lc, o), rcn = __shfl_down_sync(kFull, rc, o);
        const bool up = lane >= o, dn = lane + o < kBuckets;
        if (up) lc += lcn;
        if (dn) rc += rcn;
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            const int ln = __shfl_up_sync(kFull, l[d], o), rn = __shfl_down_sync(kFull, r[d], o);
            if (up) l[d] = d < 3 ? min(l[d], ln) : max(l[d], ln);
            if (dn) r[d] = d < 3 ? min(r[d], rn) : max(r[d], rn);
        }
    }
    rc = __shfl_down_sync(kFull, rc, 1);
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        lb[d] = kfloat(l[d]);
        rb[d] = kfloat(__shfl_down_sync(kFull, r[d], 1));
    }
    float h = 0.0f;
    if (lane < kBuckets - 1)
        h = 0.125f + ((float)lc * surface_area(lb, lb + 3) + (float)rc * surface_area(rb, rb + 3)) / outer;
    const bool ok = lane < kBuckets - 1 && h < FLT_MAX;
    const int key = ok ? fkey(h) : 0x7fffffff;
    const int best = __reduce_min_sync(kFull, key);
    const unsigned win = __ballot_sync(kFull, ok && key == best);
    return win ? __ffs(win) - 1 : -1;
}

// ---------------------------------------------------------------- phase 1: big ranges
__global__ void k_begin(Ctrl *c, Task *t0, Range *r0, Chunk *chunks, int n, int32_t *small_at,
                        int32_t *small_level) {
    const int i = threadIdx.x;
    const int nch = n > kSmall ? (n + kChunk - 1) / kChunk : 0;
    if (i == 0) {
        memset(c, 0, sizeof(Ctrl));
        if (n > kSmall) {
            c->tasks[0] = 1;
            c->chunks[0] = nch;
            *r0 = Range{0, n, 0, nch};
        } else {
            small_at[0] = n;  // a subtree of n leaves at level 0
            small_level[0] = 0;
        }
    }
    if (i < 32) clear_task(*t0, i);
    for (int k = i; k < nch; k += blockDim.x) chunks[k] = Chunk{0, k * kChunk, min(n, (k + 1) * kChunk), 0};
}

// Warp sums of 12 bound keys, then one shared atomic per warp and key.
__device__ __forceinline__ void add_bounds(int *skeys, const int (&k)[12]) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 12; ++j) {
        const int v = (j % 6) < 3 ? __reduce_min_sync(kFull, k[j]) : __reduce_max_sync(kFull, k[j]);
        if (lane == j) {
            if ((j % 6) < 3) atomicMin(skeys + j, v);
            else atomicMax(skeys + j, v);
        }
    }
}
__device__ __forceinline__ void leaf_bounds(int (&k)[12], const Leaf &l) {
    const float3 c = centroid(l);
    const int v[9] = {fkey(c.x), fkey(c.y), fkey(c.z), fkey(l.a.x), fkey(l.a.y), fkey(l.a.z),
                      fkey(l.b.x), fkey(l.b.y), fkey(l.b.z)};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        k[d] = min(k[d], v[d]);
        k[3 + d] = max(k[3 + d], v[d]);
        k[6 + d] = min(k[6 + d], v[3 + d]);
        k[9 + d] = max(k[9 + d], v[6 + d]);
    }
}
__device__ __forceinline__ void empty_bounds(int (&k)[12]) {
#pragma unroll
    for (int j = 0; j < 12; ++j) k[j] = (j % 6) < 3 ? kKeyMax : kKeyMin;
}

__global__ void __launch_bounds__(kBlock) k_leaves(const float *xyz, int n, Leaf *leaves, rg_triangle *tris,
                                                   Task *root) {
    __shared__ int skeys[12];
    if (threadIdx.x < 12) skeys[threadIdx.x] = (threadIdx.x % 6) < 3 ? kKeyMax : kKeyMin;
    __syncthreads();
    int k[12];
    empty_bounds(k);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float p[3][3];
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int d = 0; d < 3; ++d) p[v][d] = __fadd_rn(xyz[9 * (size_t)i + 3 * v + d], 0.0f);  // -0 -> +0
        float lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = nvmin(nvmin(p[0][d], p[1][d]), p[2][d]);
            hi[d] = nvmax(nvmax(p[0][d], p[1][d]), p[2][d]);
        }
        Leaf l;
        l.a = make_float4(lo[0], lo[1], lo[2], __int_as_float(i));
        l.b = make_float4(hi[0], hi[1], hi[2], 0.0f);
        leaves[i] = l;
        float4 *t = reinterpret_cast<float4 *>(tris + i);
#pragma unroll
        for (int v = 0; v < 3; ++v) t[v] = make_float4(p[v][0], p[v][1], p[v][2], 1.0f);
        leaf_bounds(k, l);
    }
    if (n > kSmall) {  // the root's bounds
        add_bounds(skeys, k);
        __syncthreads();
        if (threadIdx.x < 12) {
            if ((threadIdx.x % 6) < 3) atomicMin(root->keys + threadIdx.x, skeys[threadIdx.x]);
            else atomicMax(root->keys + threadIdx.x, skeys[threadIdx.x]);
        }
    }
}

// The buckets of every range.  A warp gathers a bucket's box over its lanes'
// leaves (four each) by warp reductions, so that a bucket costs six shared
// atomics a warp however many leaves it has: with one shared atomic per leaf
// and bound the leaves of one bucket serialise (24.6 against 16.3 us a level
// at 1.05M leaves).
__global__ void __launch_bounds__(kBlock) k_bucket(const Ctrl *c, int par, Task *ts, const Chunk *chunks,
                                                   const Leaf *leaves, uint8_t *bucket, int32_t *chunk_counts) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kPer = kChunk / kBlock;
    __shared__ int scount[kBuckets], skeys[kBuckets][6];
    const int nch = c->chunks[par], lane = threadIdx.x & 31;
    for (int ci = blockIdx.x; ci < nch; ci += gridDim.x) {
        const Chunk ch = chunks[ci];
        Task &s = ts[ch.task];
        if (threadIdx.x < kBuckets) scount[threadIdx.x] = 0;
        if (threadIdx.x < kBuckets * 6)
            skeys[threadIdx.x / 6][threadIdx.x % 6] = (threadIdx.x % 6) < 3 ? kKeyMax : kKeyMin;
        int k[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) k[j] = s.keys[j];
        const Axis ax = pick_axis(k);
        __syncthreads();
        int key[kPer][6], b[kPer];
        unsigned present = 0u;
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int p = ch.beg + e * kBlock + threadIdx.x;
            b[e] = -1;
            if (p < ch.end) {
                const Leaf l = leaves[p];
                b[e] = bucket_of(axis_of(centroid(l), ax.dim), ax.cmin, ax.range, ax.undefined);
                bucket[p] = (uint8_t)b[e];
                present |= 1u << b[e];
                key[e][0] = fkey(l.a.x); key[e][1] = fkey(l.a.y); key[e][2] = fkey(l.a.z);
                key[e][3] = fkey(l.b.x); key[e][4] = fkey(l.b.y); key[e][5] = fkey(l.b.z);
            }
        }
        for (unsigned m = __reduce_or_sync(kFull, present); m != 0u; m &= m - 1u) {
            const int q = __ffs(m) - 1;
            int cnt = 0, v[6], mine = 0;
#pragma unroll
            for (int d = 0; d < 6; ++d) v[d] = d < 3 ? kKeyMax : kKeyMin;
#pragma unroll
            for (int e = 0; e < kPer; ++e)
                if (b[e] == q) {
                    ++cnt;
#pragma unroll
                    for (int d = 0; d < 6; ++d) v[d] = d < 3 ? min(v[d], key[e][d]) : max(v[d], key[e][d]);
                }
            cnt = __reduce_add_sync(kFull, cnt);
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                const int r = d < 3 ? __reduce_min_sync(kFull, v[d]) : __reduce_max_sync(kFull, v[d]);
                if (lane == d) mine = r;
            }
            if (lane < 3) atomicMin(&skeys[q][lane], mine);
            else if (lane < 6) atomicMax(&skeys[q][lane], mine);
            else if (lane == 6) atomicAdd(&scount[q], cnt);
        }
        __syncthreads();
        const int i = threadIdx.x;
        if (i < kBuckets) {
            chunk_counts[(size_t)ci * kBuckets + i] = scount[i];
            if (scount[i]) atomicAdd(&s.bcount[i], scount[i]);
        }
        if (i < kBuckets * 6 && scount[i / 6]) {
            const int v = skeys[i / 6][i % 6];
            if ((i % 6) < 3) atomicMin(&s.bkeys[i / 6][i % 6], v);
            else atomicMax(&s.bkeys[i / 6][i % 6], v);
        }
        __syncthreads();
    }
}

// One warp per range: the split, the left leaves before each of its chunks,
// and its record; and the boxes of the previous level's median splits, whose
// halves are known only now (ts null: only those).
__global__ void __launch_bounds__(128) k_sah(Ctrl *c, int par, int level, Task *ts, const Range *ranges,
                                             Split *splits, Chunk *chunks, const int32_t *chunk_counts,
                                             const Task *prev, const Split *prev_splits, Rec *rec) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int first = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (prev)
        for (int t = first; t < c->tasks[1 - par]; t += warps)
            if (prev[t].fallback && lane < 12) rec[prev_splits[t].pivot - 1].box[lane] = kfloat(prev[t].hkeys[lane]);
    for (int t = first; ts && t < c->tasks[par]; t += warps) {
        Task &s = ts[t];
        const Range rg = ranges[t];
        int k[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) k[j] = s.keys[j];
        const Axis ax = pick_axis(k);
        int key6[6], cnt = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) key6[d] = d < 3 ? kKeyMax : kKeyMin;
        if (lane < kBuckets) {
            cnt = s.bcount[lane];
#pragma unroll
            for (int d = 0; d < 6; ++d) key6[d] = s.bkeys[lane][d];
        }
        float lb[6], rb[6];
        int lc;
        const int win = sah_warp(lane, cnt, key6, ax.outer, lb, rb, lc);
        const int opt = win < 0 ? 0 : win;
        const int nl = __shfl_sync(kFull, lc, opt);
        const int fallback = (nl == 0 || nl == rg.end - rg.beg || win < 0) ? 1 : 0;
        const int pivot = fallback ? (rg.beg + rg.end) / 2 : rg.beg + nl;
        Rec &r = rec[pivot - 1];
        if (lane == opt) {
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                r.box[j] = lb[j];
                r.box[6 + j] = rb[j];
            }
        }
        if (lane == 0) {
            s.opt = opt;
            s.nl = nl;
            s.fallback = fallback;
            splits[t].pivot = pivot;
            r.l = rg.beg;
            r.r = rg.end;
            r.level = level;
            r.rank = t;
            if (ax.undefined || win < 0) atomicOr(&c->undefined, 1);
        }
        // left leaves before each chunk
        int run = 0;
        for (int base = 0; base < rg.chunks; base += 32) {
            int v = 0;
            if (base + lane < rg.chunks)
                for (int b = 0; b <= opt; ++b) v += chunk_counts[(size_t)(rg.chunk0 + base + lane) * kBuckets + b];
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            if (base + lane < rg.chunks) chunks[rg.chunk0 + base + lane].left = run + incl - v;
            run += __shfl_sync(kFull, incl, 31);
        }
    }
}

// Block-wide exclusive scan of two counts per thread (1024 threads).
__device__ __forceinline__ void scan2(int &a, int &b, int &ta, int &tb, int2 *warp_tot) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ya = __shfl_up_sync(kFull, ia, o), yb = __shfl_up_sync(kFull, ib, o);
        if (lane >= o) {
            ia += ya;
            ib += yb;
        }
    }
    __syncthreads();  // the previous round's totals are read
    if (lane == 31) warp_tot[warp] = make_int2(ia, ib);
    __syncthreads();
    if (warp == 0) {
        int2 w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(kFull, w.x, o), yb = __shfl_up_sync(kFull, w.y, o);
            if (lane >= o) {
                w.x += ya;
                w.y += yb;
            }
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    const int2 before = warp > 0 ? warp_tot[warp - 1] : make_int2(0, 0);
    ta = warp_tot[31].x;
    tb = warp_tot[31].y;
    a = before.x + ia - a;
    b = before.y + ib - b;
}

// The next level's ranges in position order (one block: only the scan; their
// chunks and empty statistics are written by k_part); ranges of 2 to kSmall
// leaves are marked at their first position.
__global__ void __launch_bounds__(1024) k_next(Ctrl *c, int par, int level, const Range *ranges, Split *splits,
                                               Range *next, int32_t *small_at, int32_t *small_level,
                                               int32_t *big_slot, int32_t *level_big) {
    __shared__ int2 warp_tot[32];
    const int T = c->tasks[par];
    const int bigs = c->bigs;
    int nt = 0, nc = 0;
    for (int base = 0; base < T; base += 1024) {
        const int t = base + threadIdx.x;
        int cnt = 0, cch = 0;
        int bg[2] = {0, 0}, en[2] = {0, 0};
        if (t < T) {
            const Range s = ranges[t];
            bg[0] = s.beg;
            en[0] = bg[1] = splits[t].pivot;
            en[1] = s.end;
            big_slot[bigs + t] = bg[1] - 1;
            for (int k = 0; k < 2; ++k) {
                const int sz = en[k] - bg[k];
                if (sz > kSmall) {
                    ++cnt;
                    cch += (sz + kChunk - 1) / kChunk;
                } else if (sz >= 2) {
                    small_at[bg[k]] = sz;
                    small_level[bg[k]] = level + 1;
                }
            }
        }
        int at = cnt, ac = cch, tt, tc;
        scan2(at, ac, tt, tc, warp_tot);
        at += nt;
        ac += nc;
        if (t < T) {
            int child[2] = {-1, -1};
            for (int k = 0; k < 2; ++k) {
                const int sz = en[k] - bg[k];
                if (sz <= kSmall) continue;
                const int nch = (sz + kChunk - 1) / kChunk;
                next[at] = Range{bg[k], en[k], ac, nch};
                child[k] = at++;
                ac += nch;
            }
            splits[t] = Split{bg[1], {child[0], child[1]}, 0};
        }
        nt += tt;
        nc += tc;
    }
    if (threadIdx.x == 0) {
        c->tasks[1 - par] = nt;
        c->chunks[1 - par] = nc;
        c->bigs = bigs + T;
        level_big[level] = bigs;
        level_big[level + 1] = bigs + T;
        if (T > 0) c->max_level = level;
    }
}

// Every leaf's left count before it (bit 31: it is a left leaf itself), and
// the stable partition: side[beg + k] = position of the k-th left leaf,
// side[beg + nL + k] that of the k-th right one.  First the next level's
// chunk list and empty statistics, one warp per range.
__global__ void __launch_bounds__(kBlock) k_part(const Ctrl *c, int par, const Task *ts, const Range *ranges,
                                                 const Chunk *chunks, const uint8_t *bucket, uint32_t *lefts,
                                                 int32_t *side, Task *next, const Range *next_ranges,
                                                 Chunk *next_chunks) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kPer = kChunk / kBlock;
    __shared__ int warp_tot[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = blockIdx.x * (kBlock / 32) + warp; t < c->tasks[1 - par]; t += gridDim.x * (kBlock / 32)) {
        const Range r = next_ranges[t];
        clear_task(next[t], lane);
        for (int q = lane; q < r.chunks; q += 32)
            next_chunks[r.chunk0 + q] = Chunk{t, r.beg + q * kChunk, min(r.end, r.beg + (q + 1) * kChunk), 0};
    }
    const int nch = c->chunks[par];
    for (int ci = blockIdx.x; ci < nch; ci += gridDim.x) {
        const Chunk ch = chunks[ci];
        const Task &s = ts[ch.task];
        const int beg = ranges[ch.task].beg, nl = s.nl, opt = s.opt;
        const int p0 = ch.beg + threadIdx.x * kPer;
        int f[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            f[k] = p0 + k < ch.end && bucket[p0 + k] <= opt ? 1 : 0;
            sum += f[k];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        int run = ch.left + incl - sum;
        for (int w = 0; w < warp; ++w) run += warp_tot[w];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int p = p0 + k;
            if (p < ch.end) {
                lefts[p] = (uint32_t)run | ((uint32_t)f[k] << 31);
                side[f[k] ? beg + run : beg + nl + (p - beg - run)] = p;
                run += f[k];
            }
        }
        __syncthreads();
    }
}

// Every place takes its leaf (see the head of the file), and the bounds of
// both halves are gathered: for the next level's big ranges, and for the
// record of a median split.
__global__ void __launch_bounds__(kBlock) k_move(const Ctrl *c, int par, Task *ts, const Range *ranges,
                                                 const Split *splits, Task *next, const Chunk *chunks,
                                                 const uint32_t *lefts, const int32_t *side, const Leaf *in,
                                                 Leaf *out) {
    __shared__ int skeys[2][12];
    const int nch = c->chunks[par];
    for (int ci = blockIdx.x; ci < nch; ci += gridDim.x) {
        const Chunk ch = chunks[ci];
        Task &s = ts[ch.task];
        const Split sp = splits[ch.task];
        const int beg = ranges[ch.task].beg, nl = s.nl, pivot = sp.pivot;
        const bool fb = s.fallback != 0;
        if (threadIdx.x < 24) skeys[threadIdx.x / 12][threadIdx.x % 12] = (threadIdx.x % 6) < 3 ? kKeyMax : kKeyMin;
        __syncthreads();
        // the halves this chunk holds leaves of, where their bounds are wanted
        const bool want[2] = {ch.beg < pivot && (fb || sp.child[0] >= 0), ch.end > pivot && (fb || sp.child[1] >= 0)};
        int k0[12], k1[12];
        empty_bounds(k0);
        empty_bounds(k1);
        for (int q = ch.beg + threadIdx.x; q < ch.end; q += kBlock) {
            int p;
            if (q - beg < nl) {
                p = side[q];
            } else {
                p = q;
                for (uint32_t e = lefts[p]; e >> 31; e = lefts[p]) {
                    const int r = p - beg - (int)(e & 0x7fffffffu);  // right leaves before p: > 0, as q >= beg + nL
                    const int run = side[beg + nl + r - 1] + 1;      // first left leaf of p's run
                    p -= r * ((p - run) / r + 1);
                }
            }
            const Leaf l = in[p];
            out[q] = l;
            if (q < pivot) {
                if (want[0]) leaf_bounds(k0, l);
            } else {
                if (want[1]) leaf_bounds(k1, l);
            }
        }
        if (want[0]) add_bounds(skeys[0], k0);
        if (want[1]) add_bounds(skeys[1], k1);
        __syncthreads();
        if (threadIdx.x < 24) {
            const int h = threadIdx.x / 12, j = threadIdx.x % 12, v = skeys[h][j];
            if (h ? want[1] : want[0]) {
                const bool mn = (j % 6) < 3;
                const int child = h ? sp.child[1] : sp.child[0];
                if (child >= 0) {
                    if (mn) atomicMin(&next[child].keys[j], v);
                    else atomicMax(&next[child].keys[j], v);
                }
                if (fb && j >= 6) {
                    if (mn) atomicMin(&s.hkeys[6 * h + j - 6], v);
                    else atomicMax(&s.hkeys[6 * h + j - 6], v);
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- phase 2: subtrees
__global__ void k_small_flags(const int32_t *small_at, int n, int32_t *flag) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) flag[p] = small_at[p] != 0 ? 1 : 0;
}
__global__ void k_small_list(Ctrl *c, const int32_t *small_at, const int32_t *small_level, const int32_t *scan, int n,
                             Subtree *list) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) c->subtrees = scan[n];
    if (p < n && small_at[p] != 0) list[scan[p]] = Subtree{p, p + small_at[p], small_level[p]};
}

constexpr int kSubWarps = 4;  // warps (subtrees) per block

// One warp per subtree: the reference's breadth-first build over its leaves,
// from shared memory.  counts[level * U + t] receives the subtree's nodes of
// each level; levels beyond `cap` are only reported (max_level).
__global__ void __launch_bounds__(32 * kSubWarps) k_subtrees(Ctrl *c, const Subtree *list, int U, const Leaf *la,
                                                             const Leaf *lb_, Rec *rec, int32_t *counts, int cap) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ float s_lo[kSubWarps][3][kSmall], s_hi[kSubWarps][3][kSmall];
    __shared__ int s_geom[kSubWarps][kSmall];
    __shared__ uint8_t s_idx[kSubWarps][2][kSmall];     // leaf order, and the partition's output
    __shared__ uint8_t s_left[kSubWarps][kSmall];       // left count before a place, bit 7: a left leaf
    __shared__ uint8_t s_qb[kSubWarps][kSmall], s_qe[kSubWarps][kSmall];  // node queue: leaf range
    __shared__ int s_bcount[kSubWarps][kBuckets], s_bkeys[kSubWarps][kBuckets][6];
    static_assert(kSmall <= 128, "places and counts are bytes with a flag bit");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x * kSubWarps + w;
    if (t >= U) return;
    const Subtree st = list[t];
    const int m = st.end - st.beg;
    const Leaf *src = (st.level & 1) ? lb_ : la;  // the buffer its last move wrote
    float(*lo)[kSmall] = s_lo[w], (*hi)[kSmall] = s_hi[w];
    int *geom = s_geom[w];
    uint8_t *idx = s_idx[w][0], *idx2 = s_idx[w][1], *left = s_left[w], *qb = s_qb[w], *qe = s_qe[w];
    int *bcount = s_bcount[w], (*bkeys)[6] = s_bkeys[w];
    for (int k = lane; k < m; k += 32) {
        const Leaf l = src[st.beg + k];
        lo[0][k] = l.a.x; lo[1][k] = l.a.y; lo[2][k] = l.a.z;
        hi[0][k] = l.b.x; hi[1][k] = l.b.y; hi[2][k] = l.b.z;
        geom[k] = __float_as_int(l.a.w);
        idx[k] = (uint8_t)k;
    }
    if (lane == 0) {
        qb[0] = 0;
        qe[0] = (uint8_t)m;
    }
    __syncwarp();
    int tail = 1, level = st.level, level_start = 0, next_start = 1, undefined = 0;
    for (int i = 0; i < tail; ++i) {
        if (i == next_start) {
            if (lane == 0 && level < cap) counts[(size_t)level * U + t] = next_start - level_start;
            ++level;
            level_start = i;
            next_start = tail;
        }
        const int beg = qb[i], end = qe[i], sz = end - beg;
        Rec &r = rec[st.beg + i];
        if (sz == 2) {
            if (lane < 2) {
                const int e = idx[beg + lane];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    r.box[6 * lane + d] = lo[d][e];
                    r.box[6 * lane + 3 + d] = hi[d][e];
                }
                if (lane == 0) {
                    r.l = ~geom[e];
                    r.level = level;
                    r.rank = i - level_start;
                } else {
                    r.r = ~geom[e];
                }
            }
            continue;
        }
        // bounds of the range
        int k[12];
        empty_bounds(k);
        for (int j = beg + lane; j < end; j += 32) {
            const int e = idx[j];
            Leaf l;
            l.a = make_float4(lo[0][e], lo[1][e], lo[2][e], 0.0f);
            l.b = make_float4(hi[0][e], hi[1][e], hi[2][e], 0.0f);
            leaf_bounds(k, l);
        }
#pragma unroll
        for (int j = 0; j < 12; ++j)
            k[j] = (j % 6) < 3 ? __reduce_min_sync(kFull, k[j]) : __reduce_max_sync(kFull, k[j]);
        const Axis ax = pick_axis(k);
        if (lane < kBuckets) bcount[lane] = 0;
        for (int j = lane; j < kBuckets * 6; j += 32) bkeys[j / 6][j % 6] = (j % 6) < 3 ? kKeyMax : kKeyMin;
        __syncwarp();
        // buckets; a leaf's bucket stays in idx2 until the split is known
        for (int j = beg + lane; j < end; j += 32) {
            const int e = idx[j];
            const float cd = 0.5f * (lo[ax.dim][e] + hi[ax.dim][e]);
            const int b = bucket_of(cd, ax.cmin, ax.range, ax.undefined);
            left[j] = (uint8_t)b;
            atomicAdd(&bcount[b], 1);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                atomicMin(&bkeys[b][d], fkey(lo[d][e]));
                atomicMax(&bkeys[b][3 + d], fkey(hi[d][e]));
            }
        }
        __syncwarp();
        int key6[6], cnt = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) key6[d] = d < 3 ? kKeyMax : kKeyMin;
        if (lane < kBuckets) {
            cnt = bcount[lane];
#pragma unroll
            for (int d = 0; d < 6; ++d) key6[d] = bkeys[lane][d];
        }
        float lbx[6], rbx[6];
        int lc;
        const int win = sah_warp(lane, cnt, key6, ax.outer, lbx, rbx, lc);
        const int opt = win < 0 ? 0 : win;
        const int nl = __shfl_sync(kFull, lc, opt);
        const bool fallback = nl == 0 || nl == sz || win < 0;
        // (beg + end) / 2 over positions of the whole leaf array, as the reference divides
        const int pivot = fallback ? (2 * st.beg + beg + end) / 2 - st.beg : beg + nl;
        if (ax.undefined || win < 0) undefined = 1;
        // the partition
        int run = 0;
        for (int base = beg; base < end; base += 32) {
            const int j = base + lane;
            const bool f = j < end && left[j] <= opt;
            const unsigned mask = __ballot_sync(kFull, f);
            const int l = run + __popc(mask & ((1u << lane) - 1u));
            if (f) idx2[beg + l] = idx[j];
            if (j < end) left[j] = (uint8_t)(l | (f ? 128 : 0));
            run += __popc(mask);
        }
        __syncwarp();
        for (int q = beg + nl + lane; q < end; q += 32) {
            int p = q;
            while (left[p] & 128) p = beg + (left[p] & 127);
            idx2[q] = idx[p];
        }
        __syncwarp();
        for (int j = beg + lane; j < end; j += 32) idx[j] = idx2[j];
        __syncwarp();
        if (fallback) {  // the halves' boxes
            int h[12];
            empty_bounds(h);
            for (int j = beg + lane; j < end; j += 32) {
                const int e = idx[j];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if (j < pivot) {
                        h[d] = min(h[d], fkey(lo[d][e]));
                        h[3 + d] = max(h[3 + d], fkey(hi[d][e]));
                    } else {
                        h[6 + d] = min(h[6 + d], fkey(lo[d][e]));
                        h[9 + d] = max(h[9 + d], fkey(hi[d][e]));
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 12; ++j) {
                const int v = (j % 6) < 3 ? __reduce_min_sync(kFull, h[j]) : __reduce_max_sync(kFull, h[j]);
                if (lane == 0) r.box[j] = kfloat(v);
            }
        } else if (lane == opt) {
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                r.box[j] = lbx[j];
                r.box[6 + j] = rbx[j];
            }
        }
        const int szl = pivot - beg, szr = end - pivot;
        const int cl = tail, cr = tail + (szl > 1 ? 1 : 0);
        if (lane == 0) {
            r.l = szl > 1 ? cl - next_start : ~geom[idx[beg]];
            r.r = szr > 1 ? cr - next_start : ~geom[idx[pivot]];
            r.level = level;
            r.rank = i - level_start;
            if (szl > 1) {
                qb[cl] = (uint8_t)beg;
                qe[cl] = (uint8_t)pivot;
            }
            if (szr > 1) {
                qb[cr] = (uint8_t)pivot;
                qe[cr] = (uint8_t)end;
            }
        }
        tail = cr + (szr > 1 ? 1 : 0);
        __syncwarp();
    }
    if (lane == 0) {
        if (level < cap) counts[(size_t)level * U + t] = tail - level_start;
        atomicMax(&c->max_level, level);
        if (undefined) atomicOr(&c->undefined, 1);
    }
}

// ---------------------------------------------------------------- phase 3: numbering
// counts[level][0..U) -> exclusive prefix over the subtrees, the total in
// totals[level]; one block per level.
__global__ void __launch_bounds__(1024) k_level_scan(const Ctrl *c, int32_t *counts, int U, int32_t *totals) {
    __shared__ int2 warp_tot[32];
    const int L = blockIdx.x;
    if (L > c->max_level) return;
    int32_t *row = counts + (size_t)L * U;
    int run = 0;
    for (int base = 0; base < U; base += 1024) {
        const int t = base + threadIdx.x;
        int v = t < U ? row[t] : 0, z = 0, tot, tz;
        scan2(v, z, tot, tz, warp_tot);
        if (t < U) row[t] = run + v;
        run += tot;
    }
    if (threadIdx.x == 0) totals[L] = run;
}
// base[L] = nodes of the levels above L (one thread: a level is a node)
__global__ void k_level_base(const Ctrl *c, const int32_t *totals, const int32_t *level_big, int big_levels, int cap,
                             int32_t *base) {
    if (c->max_level >= cap) return;  // the host repeats with more levels
    int run = 0;
    for (int L = 0; L <= c->max_level; ++L) {
        base[L] = run;
        run += totals[L] + (L < big_levels ? level_big[L + 1] - level_big[L] : 0);
    }
    base[c->max_level + 1] = run;
}

__device__ __forceinline__ void put_node(rg_aabb_tree_node *nodes, int id, const Rec &r, int left, int right) {
    float4 *d = reinterpret_cast<float4 *>(nodes + id);
#pragma unroll
    for (int k = 0; k < 4; ++k) d[k] = make_float4(r.box[3 * k], r.box[3 * k + 1], r.box[3 * k + 2], 1.0f);
    d[4] = make_float4(__int_as_float(left), __int_as_float(right), 0.0f, 0.0f);
}
struct Numbers {
    const int32_t *base, *counts, *level_big, *big_slot, *before;  // before[p]: subtrees whose first leaf is before p
    const Rec *rec;
    int U, big_levels;
};
// big ranges of level L that begin before position p
__device__ __forceinline__ int bigs_before(const Numbers &nb, int L, int p) {
    if (L >= nb.big_levels) return 0;
    int lo = nb.level_big[L], hi = nb.level_big[L + 1];
    const int first = lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (nb.rec[nb.big_slot[mid]].l < p) lo = mid + 1;
        else hi = mid;
    }
    return lo - first;
}
__device__ __forceinline__ int subtree_base(const Numbers &nb, int L, int t, int beg) {
    return nb.base[L] + bigs_before(nb, L, beg) + nb.counts[(size_t)L * nb.U + t];
}
// The number of the node over [beg, end) at level L, or the leaf's link.
__device__ __forceinline__ int link_of(const Numbers &nb, int L, int beg, int end, int big, const Leaf *leaves) {
    if (end - beg == 1) return ~__float_as_int(leaves[beg].a.w);
    const int t = nb.before[beg];
    if (end - beg <= kSmall) return subtree_base(nb, L, t, beg);
    return nb.base[L] + big + (t < nb.U ? nb.counts[(size_t)L * nb.U + t] : nb.base[L + 1] - nb.base[L] -
                               (nb.level_big[L + 1] - nb.level_big[L]));
}
__global__ void __launch_bounds__(128) k_emit_big(const Ctrl *c, int cap, int bigs, Numbers nb, const Leaf *la, const Leaf *lb,
                                                  rg_aabb_tree_node *nodes) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= bigs || c->max_level >= cap) return;
    const int slot = nb.big_slot[k];
    const Rec &r = nb.rec[slot];
    const int L = r.level, pivot = slot + 1;
    const int id = link_of(nb, L, r.l, r.r, r.rank, nullptr);
    const Leaf *lv = ((L + 1) & 1) ? lb : la;
    const int bl = pivot - r.l > kSmall ? bigs_before(nb, L + 1, r.l) : 0;
    const int br = r.r - pivot > kSmall ? bigs_before(nb, L + 1, pivot) : 0;
    const int left = link_of(nb, L + 1, r.l, pivot, bl, lv), right = link_of(nb, L + 1, pivot, r.r, br, lv);
    put_node(nodes, id, r, left, right);
}
__global__ void __launch_bounds__(128) k_emit_subtrees(const Ctrl *c, int cap, const Subtree *list, Numbers nb,
                                                       rg_aabb_tree_node *nodes) {
    const int lane = threadIdx.x & 31;
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= nb.U || c->max_level >= cap) return;
    const Subtree st = list[t];
    for (int i = lane; i < st.end - st.beg - 1; i += 32) {
        const Rec r = nb.rec[st.beg + i];
        const int id = subtree_base(nb, r.level, t, st.beg) + r.rank;
        int left = r.l, right = r.r;
        if (left >= 0 || right >= 0) {
            const int b = subtree_base(nb, r.level + 1, t, st.beg);
            if (left >= 0) left += b;
            if (right >= 0) right += b;
        }
        put_node(nodes, id, r, left, right);
    }
}

// ---- exclusive scan of n int32 flags into out[0..n] (out[n] = total), n <= 4M
constexpr int kScanThreads = 256, kScanPer = 8, kScanBlock = kScanThreads * kScanPer;

__global__ void k_scan_block(const int32_t *in, int n, int32_t *out, int32_t *block_sums) {
    __shared__ int32_t warp_sums[kScanThreads / 32];
    const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
    int32_t v[kScanPer], s = 0;
    for (int k = 0; k < kScanPer; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t incl = s;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int32_t w = lane < kScanThreads / 32 ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    int32_t run = incl - s + (warp > 0 ? warp_sums[warp - 1] : 0);
    for (int k = 0; k < kScanPer; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == kScanThreads - 1) block_sums[blockIdx.x] = run;
}
__global__ void k_scan_add(int32_t *out, int n, const int32_t *block_offsets, const int32_t *block_sums, int nb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += block_offsets[i / kScanBlock];
    else if (i == n) out[n] = block_offsets[nb - 1] + block_sums[nb - 1];
}

// Bytes of workspace in order; every piece 256-byte aligned.
struct Carve {
    unsigned char *base = nullptr;
    size_t at = 0;
    template <typename T> T *take(size_t count) {
        T *p = base ? reinterpret_cast<T *>(base + at) : nullptr;
        at += (count * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
};
struct Work {
    Leaf *leaves[2];
    Rec *rec;
    Task *tasks[2];
    Range *ranges[2];
    Split *splits[2];
    Chunk *chunks[2];
    uint8_t *bucket;
    uint32_t *lefts;
    int32_t *side, *chunk_counts, *small_at, *small_level, *flag, *before, *big_slot, *level_big, *base, *totals, *sums,
        *offs;
    Subtree *list;
    Ctrl *ctrl;
    int max_tasks, max_chunks;
    explicit Work(Carve &c, int n) {
        const size_t nn = (size_t)n;
        max_tasks = n / (kSmall + 1) + 1;  // a level's big ranges are disjoint
        max_chunks = n / kChunk + max_tasks + 1;
        for (int k = 0; k < 2; ++k) {
            leaves[k] = c.take<Leaf>(nn);
            tasks[k] = c.take<Task>((size_t)max_tasks);
            ranges[k] = c.take<Range>((size_t)max_tasks);
            splits[k] = c.take<Split>((size_t)max_tasks);
            chunks[k] = c.take<Chunk>((size_t)max_chunks);
        }
        rec = c.take<Rec>(nn);
        bucket = c.take<uint8_t>(nn);
        lefts = c.take<uint32_t>(nn);
        side = c.take<int32_t>(nn);
        chunk_counts = c.take<int32_t>((size_t)max_chunks * kBuckets);
        small_at = c.take<int32_t>(nn);
        small_level = c.take<int32_t>(nn);
        flag = c.take<int32_t>(nn);
        before = c.take<int32_t>(nn + 1);
        big_slot = c.take<int32_t>(nn);
        level_big = c.take<int32_t>(nn + 2);
        base = c.take<int32_t>(nn + 2);
        totals = c.take<int32_t>(nn + 2);
        const size_t blocks = (nn + kScanBlock - 1) / kScanBlock;
        sums = c.take<int32_t>(blocks);
        offs = c.take<int32_t>(blocks + 1);
        list = c.take<Subtree>(nn / 2 + 1);
        ctrl = c.take<Ctrl>(1);
    }
};

cudaError_t scan_flags(const Work &w, int n, cudaStream_t st) {
    const int nb = (n + kScanBlock - 1) / kScanBlock;
    k_scan_block<<<nb, kScanThreads, 0, st>>>(w.flag, n, w.before, w.sums);
    k_scan_block<<<1, kScanThreads, 0, st>>>(w.sums, nb, w.offs, w.totals);
    k_scan_add<<<(n + 256) / 256, 256, 0, st>>>(w.before, n, w.offs, w.sums, nb);
    return cudaGetLastError();
}

}  // namespace

// Builds the tree of n triangles (9 floats each, device) into nodes[n-1] and
// tris[n] (device), synchronously on `st`, with the context's workspace.
// Returns the node count or an RG_ERR_* code; *undefined receives whether a
// range took the reference-undefined path (coincident centroids or zero area).
static int gpu_build_bvh(rg_context *ctx, const float *xyz, int n, rg_aabb_tree_node *nodes, rg_triangle *tris,
                         int *undefined, cudaStream_t st) {
    Carve size;
    (void)Work(size, n);
    void *mem = nullptr;
    int rc = rg_internal_tree_workspace(ctx, 0, size.at, &mem);
    if (rc) return rc;
    Carve place;
    place.base = static_cast<unsigned char *>(mem);
    const Work w(place, n);
    const int gn = (n + 255) / 256;
    cudaError_t e = cudaMemsetAsync(w.small_at, 0, (size_t)n * 4, st);
    if (e != cudaSuccess) return rg_internal_fail(RG_ERR_CUDA, cudaGetErrorString(e));
    k_begin<<<1, 256, 0, st>>>(w.ctrl, w.tasks[0], w.ranges[0], w.chunks[0], n, w.small_at, w.small_level);
    k_leaves<<<gn, kBlock, 0, st>>>(xyz, n, w.leaves[0], tris, w.tasks[0]);
    // as many levels as a tree with somewhat uneven splits needs before its
    // ranges are small, then more in threes while big ranges are left
    int levels = 0, more = 0;
    while (n > kSmall && (kSmall << more) < n) ++more;
    if (n > kSmall) more += 4;
    Ctrl c{};
    for (;;) {
        for (int k = 0; k < more; ++k, ++levels) {
            const int par = levels & 1;
            const int tasks = levels < 20 && (1 << levels) < w.max_tasks ? 1 << levels : w.max_tasks;
            const int chunks = n / kChunk + tasks + 1 < w.max_chunks ? n / kChunk + tasks + 1 : w.max_chunks;
            const int gc = chunks < 152 * 8 ? chunks : 152 * 8;
            const int gw = (tasks + 3) / 4 < 152 * 8 ? (tasks + 3) / 4 : 152 * 8;
            const int nxt = 1 - par;
            Task *ts = w.tasks[par], *next = w.tasks[nxt];
            k_bucket<<<gc, kBlock, 0, st>>>(w.ctrl, par, ts, w.chunks[par], w.leaves[par], w.bucket, w.chunk_counts);
            k_sah<<<gw, 128, 0, st>>>(w.ctrl, par, levels, ts, w.ranges[par], w.splits[par], w.chunks[par],
                                      w.chunk_counts, levels > 0 ? next : nullptr, w.splits[nxt], w.rec);
            k_next<<<1, 1024, 0, st>>>(w.ctrl, par, levels, w.ranges[par], w.splits[par], w.ranges[nxt], w.small_at,
                                       w.small_level, w.big_slot, w.level_big);
            k_part<<<gc, kBlock, 0, st>>>(w.ctrl, par, ts, w.ranges[par], w.chunks[par], w.bucket, w.lefts, w.side,
                                          next, w.ranges[nxt], w.chunks[nxt]);
            k_move<<<gc, kBlock, 0, st>>>(w.ctrl, par, ts, w.ranges[par], w.splits[par], next, w.chunks[par], w.lefts,
                                          w.side, w.leaves[par], w.leaves[nxt]);
        }
        if (levels > 0)  // the last level's median splits
            k_sah<<<152, 128, 0, st>>>(w.ctrl, levels & 1, levels, nullptr, nullptr, nullptr, nullptr, nullptr,
                                       w.tasks[1 - (levels & 1)], w.splits[1 - (levels & 1)], w.rec);
        k_small_flags<<<gn, 256, 0, st>>>(w.small_at, n, w.flag);
        e = scan_flags(w, n, st);
        k_small_list<<<gn, 256, 0, st>>>(w.ctrl, w.small_at, w.small_level, w.before, n, w.list);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&c, w.ctrl, sizeof(c), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return rg_internal_fail(RG_ERR_CUDA, cudaGetErrorString(e));
        if (c.tasks[levels & 1] == 0) break;
        more = 3;
    }
    const int U = c.subtrees, bigs = c.bigs;
    // levels of the tree are known after the subtrees: a first guess of the
    // deepest, and once more in the rare case that it was too low
    int cap = levels + 24, bound = 0;
    for (;;) {
        void *cm = nullptr;
        if ((rc = rg_internal_tree_workspace(ctx, 1, (size_t)cap * (size_t)U * 4, &cm))) return rc;
        int32_t *counts = static_cast<int32_t *>(cm);
        e = cudaMemsetAsync(counts, 0, (size_t)cap * (size_t)U * 4, st);
        k_subtrees<<<(U + kSubWarps - 1) / kSubWarps, 32 * kSubWarps, 0, st>>>(w.ctrl, w.list, U, w.leaves[0],
                                                                               w.leaves[1], w.rec, counts, cap);
        k_level_scan<<<cap, 1024, 0, st>>>(w.ctrl, counts, U, w.totals);
        k_level_base<<<1, 1, 0, st>>>(w.ctrl, w.totals, w.level_big, levels, cap, w.base);
        const Numbers nb{w.base, counts, w.level_big, w.big_slot, w.before, w.rec, U, levels};
        if (bigs > 0)
            k_emit_big<<<(bigs + 127) / 128, 128, 0, st>>>(w.ctrl, cap, bigs, nb, w.leaves[0], w.leaves[1], nodes);
        k_emit_subtrees<<<(U + 3) / 4, 128, 0, st>>>(w.ctrl, cap, w.list, nb, nodes);
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&c, w.ctrl, sizeof(c), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return rg_internal_fail(RG_ERR_CUDA, cudaGetErrorString(e));
        if (c.max_level < cap) break;
        if (bound++) return rg_internal_fail(RG_ERR_CUDA, "rg_build_bvh_device: level count changed");
        cap = c.max_level + 1;
    }
    *undefined = c.undefined;
    return n - 1;
}

extern "C" int rg_build_bvh_device(rg_context *ctx, const float *tri_xyz, int32_t n_tris, rg_aabb_tree_node *nodes,
                                   rg_triangle *triangles, int32_t *ref_undefined, void *stream) {
    int device = 0;
    int rc = rg_internal_device(ctx, &device);
    if (rc) return rc;
    if (!tri_xyz || !nodes || !triangles) return rg_internal_fail(RG_ERR_INVALID_ARGUMENT, "null pointer");
    if (n_tris < 2 || n_tris > (1 << 22))
        return rg_internal_fail(RG_ERR_INVALID_ARGUMENT, "rg_build_bvh_device: 2 .. 4194304 triangles");
    if (((uintptr_t)tri_xyz & 3u) || ((uintptr_t)nodes & 15u) || ((uintptr_t)triangles & 15u))
        return rg_internal_fail(RG_ERR_INVALID_ARGUMENT, "misaligned buffer");
    int undef = 0;
    const int r = gpu_build_bvh(ctx, tri_xyz, n_tris, nodes, triangles, &undef, (cudaStream_t)stream);
    if (r < 0) return r;
    if (ref_undefined) *ref_undefined = undef;
    return r;
}
