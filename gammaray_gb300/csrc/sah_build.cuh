// The reference's SAH tree (geom/bvh.rs:182-382) built on the device for large scenes: the
// same splits and the same component order as the host build (scene_build.cpp), so the same
// hits.  Every choice of that build depends only on a node's components and their order:
//
//   * boxes and centroid bounds are minima and maxima, the bucket counts whole numbers, the
//     costs the same float expressions: exact in any order;
//   * its partition swaps matches to the front.  With k matches, p1 the first non-match, T
//     the positions of the matches after it and R = |T|, the matches keep their order at
//     the front, and the non-match at position p ends at k + pos - R, where pos starts at
//     p - p1 and steps pos = T[pos] - p1 while pos < R: every element finds its place alone
//     (sah_walk.cuh);
//   * a node whose centroids coincide is a leaf there.  Its components are halved here, as
//     the collapse halves a range, down to single ones.
//
// Nodes of more than sah_small() components are split level by level by the whole grid, four
// launches a level (k_sah_buckets, k_sah_count, k_sah_front, k_sah_back), in tiles.  A block
// then builds each smaller subtree in shared memory (k_sah_small).  The binary tree has one
// internal node per gap between neighbouring components of the final order, which is its
// index.
//
// Bound by the launches of its levels (a dozen) and the chain of each.  Creation of a scene of
// 200,000 triangles takes 1.8 ms, with the host build on 16 cores 11.6.  Coordinates that are
// not finite, and trees too deep for the level limits, are left to the host.  Positions read
// from the order are kept inside their arrays whatever they hold.
#pragma once

#include "sah_walk.cuh"

namespace gr {

namespace {

constexpr int SAH_BUCKETS = 12;
constexpr int SAH_VALUES = 13;  // per bucket: count, box lo and hi, centroid lo and hi
// Most components of a subtree that one block builds, by the scene's: a block takes its
// subtree's first levels a warp at a time, so smaller subtrees, whose splits the whole grid
// shares, end sooner, until there are so many nodes that the levels cost more.  256 / 512 /
// 1024 measured 984 / 1069 / 1137 us of scene creation for 4,100 triangles, 1356 / 1408 /
// 1541 for 20,000, 1658 / 1698 / 1830 for 102,400, 2190 / 2113 / 2159 for 200,000 and 2577 /
// 2536 / 2399 for 400,000 (with scratch from cudaMalloc).
constexpr uint32_t SAH_SMALL_FEW = 256, SAH_SMALL_MANY = 1024;
constexpr uint32_t SAH_MANY = 150000;
inline uint32_t sah_small(uint32_t n) { return n < SAH_MANY ? SAH_SMALL_FEW : SAH_SMALL_MANY; }
constexpr uint32_t SAH_TILE = 1024;
constexpr uint32_t SAH_ROOT = 0xFFFFFFFFu;
constexpr uint32_t SAH_LEVELS = 64;  // of large nodes
constexpr int SAH_WARPS = BB / 32;

struct SahCtl {
    uint32_t big[SAH_LEVELS + 1], tiles[SAH_LEVELS + 1];  // of each level
    uint32_t small;
    uint32_t excess;  // components beyond the first of every leaf of the reference's tree
    uint32_t failed;  // the host build takes over
    int root;         // index of the root's internal node
    int bounds[12];   // of all components: box lo, hi, centroid lo, hi (ordered)
};

// A large node.
struct SahNode {
    uint32_t first, count;
    uint32_t slot;   // its place in its parent's record: 2 * parent + side, or SAH_ROOT
    uint32_t range;  // its centroids coincide
    float box[6], cb[6];
};

struct SahSmall {
    uint32_t first, count, slot;
    uint32_t flags;  // bit 0: range, bit 1: which order buffer holds it
};

// One level's nodes (tables: SAH_BUCKETS x SAH_VALUES per node).
struct SahLevel {
    SahNode* nodes;
    int* tables;
    uint32_t* first_out;  // first component that does not go to the left, in the node
    uint32_t* tile0;      // a node's first tile
    uint2* tiles;         // (node, tile of the node)
};

// What all kernels of the build read and write.
struct SahView {
    SahCtl* ctl;
    const float* box;  // 6 per component
    uint32_t* order[2];
    uint8_t* bucket;      // per position
    uint32_t* moved;      // T, per position
    uint32_t* tile_left;  // matches per tile
    uint32_t* best;       // per node: last bucket of the left side
    uint32_t* left;       // per node: components of the left side
    SahSmall* small;
    float* opened;  // the internal nodes' records (Opened), 16 floats each
    uint32_t n, most_small, max_big, max_tiles, max_small;
    SahLevel level[2];
};

GR_D int sah_empty(int v) {  // value v of an empty bucket
    return v == 0 ? 0 : ((v - 1) / 3 % 2 == 0 ? ordered(FLT_MAX) : ordered(-FLT_MAX));
}
GR_D float volume6(const float* b) { return (b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2]); }
GR_D int max_extent6(const float* b) {
    const float dx = b[3] - b[0], dy = b[4] - b[1], dz = b[5] - b[2];
    return dx >= dy && dy >= dz ? 0 : (dy >= dz ? 1 : 2);
}
GR_D uint32_t sah_bucket(float c, float lo, float hi) {
    const float rel = (c - lo) / (hi - lo);
    const float f = static_cast<float>(SAH_BUCKETS) * rel;
    return f >= 0.0f ? min(static_cast<uint32_t>(SAH_BUCKETS - 1), static_cast<uint32_t>(f)) : 0u;
}

// Cost of splitting after bucket i.
GR_D float sah_cost(const int* tab, int i, const float* box) {
    float side[2][6];
    uint32_t count[2] = {0, 0};
    for (int s = 0; s < 2; ++s)
        for (int a = 0; a < 3; ++a) {
            side[s][a] = FLT_MAX;
            side[s][3 + a] = -FLT_MAX;
        }
    for (int j = 0; j < SAH_BUCKETS; ++j) {
        const int s = j <= i ? 0 : 1;
        const int* t = tab + j * SAH_VALUES;
        count[s] += static_cast<uint32_t>(t[0]);
        for (int a = 0; a < 3; ++a) {
            const float lo = unordered(t[1 + a]), hi = unordered(t[4 + a]);
            if (s == 0) {
                side[0][a] = fminf(side[0][a], lo);
                side[0][3 + a] = fmaxf(side[0][3 + a], hi);
            } else {
                side[1][a] = fminf(side[1][a], lo);
                side[1][3 + a] = fmaxf(side[1][3 + a], hi);
            }
        }
    }
    return 1.0f + (static_cast<float>(count[0]) * volume6(side[0]) + static_cast<float>(count[1]) * volume6(side[1])) /
                      volume6(box);
}

// The cheapest split of a warp's table (the first of equal ones); `cost` receives its cost.
// Every lane calls it.
GR_D uint32_t sah_best(const int* tab, const float* box, float& cost) {
    const unsigned lane = threadIdx.x & 31u;
    const float mine = lane < SAH_BUCKETS - 1 ? sah_cost(tab, static_cast<int>(lane), box) : 0.0f;
    uint32_t best = 0;
    cost = __shfl_sync(0xffffffffu, mine, 0);
    for (int i = 1; i < SAH_BUCKETS - 1; ++i) {
        const float c = __shfl_sync(0xffffffffu, mine, i);
        if (c < cost) {
            cost = c;
            best = static_cast<uint32_t>(i);
        }
    }
    return best;
}

// Adds the warp's components (in: this lane has one, in bucket b, with its box and centroid)
// to `tab`.  With ATOMIC other warps add to it too.  Every lane calls it.
template <bool ATOMIC>
GR_D void sah_add(int* tab, bool in, uint32_t b, const float* x, const float* c) {
    const unsigned all = 0xffffffffu, lane = threadIdx.x & 31u;
    for (unsigned rest = __ballot_sync(all, in); rest;) {
        const uint32_t pick = __shfl_sync(all, b, __ffs(rest) - 1);
        const bool mine = in && b == pick;
        const unsigned who = __ballot_sync(all, mine);
        rest &= ~who;
        int v = __popc(who);
        for (int a = 0; a < 3; ++a) {
            const int bl = __reduce_min_sync(all, mine ? ordered(x[a]) : 0x7FFFFFFF);
            const int bh = __reduce_max_sync(all, mine ? ordered(x[3 + a]) : static_cast<int>(0x80000000u));
            const int cl = __reduce_min_sync(all, mine ? ordered(c[a]) : 0x7FFFFFFF);
            const int ch = __reduce_max_sync(all, mine ? ordered(c[a]) : static_cast<int>(0x80000000u));
            if (lane == 1u + a) v = bl;
            if (lane == 4u + a) v = bh;
            if (lane == 7u + a) v = cl;
            if (lane == 10u + a) v = ch;
        }
        if (lane < SAH_VALUES) {
            int* t = tab + pick * SAH_VALUES + lane;
            const bool low = (lane >= 1 && lane < 4) || (lane >= 7 && lane < 10);
            if (ATOMIC) {
                if (lane == 0) atomicAdd(t, v);
                else if (low) atomicMin(t, v);
                else atomicMax(t, v);
            } else {
                *t = lane == 0 ? *t + v : (low ? min(*t, v) : max(*t, v));
            }
        }
        __syncwarp();
    }
}

GR_D void sah_load(const SahView& s, uint32_t id, float* x, float* c) {
    const float2* p = reinterpret_cast<const float2*>(s.box + 6 * static_cast<size_t>(min(id, s.n - 1)));
    const float2 a = __ldg(p), b = __ldg(p + 1), d = __ldg(p + 2);
    x[0] = a.x;
    x[1] = a.y;
    x[2] = b.x;
    x[3] = b.y;
    x[4] = d.x;
    x[5] = d.y;
    for (int q = 0; q < 3; ++q) c[q] = 0.5f * x[q] + 0.5f * x[3 + q];  // bvh.rs:26
}

// Enters a node into the next level or the small ones.  Every lane of a warp calls it.
GR_D void sah_enter(const SahView& s, uint32_t level, SahNode nd) {
    const unsigned lane = threadIdx.x & 31u;
    const int dim = max_extent6(nd.cb);
    if (nd.count > 1 && !nd.range && nd.cb[dim] == nd.cb[3 + dim]) {
        nd.range = 1;
        if (lane == 0) atomicAdd(&s.ctl->excess, nd.count - 1);
    }
    uint32_t at = 0, tile = 0;
    const uint32_t tiles = (nd.count + SAH_TILE - 1) / SAH_TILE;
    if (nd.count > s.most_small) {
        if (lane == 0) {
            at = atomicAdd(&s.ctl->big[level], 1u);
            tile = atomicAdd(&s.ctl->tiles[level], tiles);
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        const SahLevel& L = s.level[level & 1];
        if (at >= s.max_big || tile + tiles > s.max_tiles) {  // cannot be: the sizes are bounds
            if (lane == 0) atomicExch(&s.ctl->failed, 1u);
            return;
        }
        if (lane == 0) {
            L.nodes[at] = nd;
            L.first_out[at] = nd.count;
            L.tile0[at] = tile;
        }
        for (uint32_t k = lane; k < tiles; k += 32) L.tiles[tile + k] = make_uint2(at, k);
        for (uint32_t k = lane; k < SAH_BUCKETS * SAH_VALUES; k += 32)
            L.tables[at * (SAH_BUCKETS * SAH_VALUES) + k] = sah_empty(static_cast<int>(k % SAH_VALUES));
    } else if (lane == 0) {
        at = atomicAdd(&s.ctl->small, 1u);
        if (at < s.max_small) s.small[at] = SahSmall{nd.first, nd.count, nd.slot, nd.range | ((level & 1u) << 1)};
        else atomicExch(&s.ctl->failed, 1u);
    }
}

// Bounds of all components, and the first order.
__global__ void __launch_bounds__(BB) k_sah_bounds(SahView s) {
    float lo[6], hi[6];
    for (int a = 0; a < 6; ++a) {
        lo[a] = FLT_MAX;
        hi[a] = -FLT_MAX;
    }
    bool odd = false;
    for (uint32_t k = blockIdx.x * BB + threadIdx.x; k < s.n; k += gridDim.x * BB) {
        float x[6], c[3];
        sah_load(s, k, x, c);
        for (int a = 0; a < 3; ++a) {
            odd |= !isfinite(x[a]) || !isfinite(x[3 + a]) || !isfinite(c[a]);
            lo[a] = fminf(lo[a], x[a]);
            hi[a] = fmaxf(hi[a], x[3 + a]);
            lo[3 + a] = fminf(lo[3 + a], c[a]);
            hi[3 + a] = fmaxf(hi[3 + a], c[a]);
        }
        s.order[0][k] = k;
    }
    if (odd) atomicExch(&s.ctl->failed, 1u);
    for (int a = 0; a < 6; ++a) {
        const int l = __reduce_min_sync(0xffffffffu, ordered(lo[a]));
        const int h = __reduce_max_sync(0xffffffffu, ordered(hi[a]));
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(&s.ctl->bounds[a < 3 ? a : a + 3], l);
            atomicMax(&s.ctl->bounds[a < 3 ? a + 3 : a + 6], h);
        }
    }
}

// The root (one warp).
__global__ void k_sah_root(SahView s) {
    SahNode nd;
    nd.first = 0;
    nd.count = s.n;
    nd.slot = SAH_ROOT;
    nd.range = 0;
    for (int a = 0; a < 6; ++a) {
        nd.box[a] = unordered(s.ctl->bounds[a]);
        nd.cb[a] = unordered(s.ctl->bounds[6 + a]);
    }
    sah_enter(s, 0, nd);
}

// The bucket of each component of a level's nodes, and the nodes' tables.  Bound by the
// reductions of a warp's buckets (12 a bucket); one atomic per value, bucket and tile then
// reaches memory.
__global__ void __launch_bounds__(BB) k_sah_buckets(SahView s, uint32_t level) {
    __shared__ int tab[SAH_BUCKETS * SAH_VALUES];
    const SahLevel& L = s.level[level & 1];
    const uint32_t tiles = s.ctl->failed ? 0u : s.ctl->tiles[level];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint2 tile = L.tiles[t];
        const SahNode& nd = L.nodes[tile.x];
        const uint32_t first = nd.first, count = nd.count;
        const bool range = nd.range != 0;
        const int dim = max_extent6(nd.cb);
        const float lo = nd.cb[dim], hi = nd.cb[3 + dim];
        for (uint32_t k = threadIdx.x; k < SAH_BUCKETS * SAH_VALUES; k += BB)
            tab[k] = sah_empty(static_cast<int>(k % SAH_VALUES));
        __syncthreads();
        for (uint32_t e = 0; e < SAH_TILE; e += BB) {
            const uint32_t i = tile.y * SAH_TILE + e + threadIdx.x;
            const bool in = i < count;
            float x[6] = {}, c[3] = {};
            uint32_t b = 0;
            if (in) {
                sah_load(s, s.order[level & 1][first + i], x, c);
                b = range ? (i < count / 2 ? 0u : 1u) : sah_bucket(dim == 0 ? c[0] : (dim == 1 ? c[1] : c[2]), lo, hi);
                s.bucket[first + i] = static_cast<uint8_t>(b);
            }
            sah_add<true>(tab, in, b, x, c);
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < SAH_BUCKETS * SAH_VALUES; k += BB) {
            const int v = static_cast<int>(k % SAH_VALUES);
            if (tab[k - v] == 0) continue;
            int* g = L.tables + tile.x * (SAH_BUCKETS * SAH_VALUES) + k;
            if (v == 0) atomicAdd(g, tab[k]);
            else if ((v - 1) / 3 % 2 == 0) atomicMin(g, tab[k]);
            else atomicMax(g, tab[k]);
        }
        __syncthreads();
    }
}

// The split of a level's nodes, and each tile's components that go to the left.
__global__ void __launch_bounds__(BB) k_sah_count(SahView s, uint32_t level) {
    __shared__ int tab[SAH_BUCKETS * SAH_VALUES];
    __shared__ uint32_t best, matches, out;
    const SahLevel& L = s.level[level & 1];
    const uint32_t tiles = s.ctl->failed ? 0u : s.ctl->tiles[level];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint2 tile = L.tiles[t];
        const SahNode& nd = L.nodes[tile.x];
        for (uint32_t k = threadIdx.x; k < SAH_BUCKETS * SAH_VALUES; k += BB)
            tab[k] = L.tables[tile.x * (SAH_BUCKETS * SAH_VALUES) + k];
        if (threadIdx.x == 0) {
            matches = 0;
            out = nd.count;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            float cost;
            const uint32_t b = nd.range ? 0u : sah_best(tab, nd.box, cost);
            if (threadIdx.x == 0) {
                best = b;
                if (tile.y == 0) s.best[tile.x] = b;
            }
        }
        __syncthreads();
        for (uint32_t e = 0; e < SAH_TILE; e += BB) {
            const uint32_t i = tile.y * SAH_TILE + e + threadIdx.x;
            const bool in = i < nd.count, left = in && s.bucket[nd.first + i] <= best;
            const unsigned m = __ballot_sync(0xffffffffu, left);
            const uint32_t o = __reduce_min_sync(0xffffffffu, in && !left ? i : 0xFFFFFFFFu);
            if ((threadIdx.x & 31u) == 0) {
                atomicAdd(&matches, static_cast<uint32_t>(__popc(m)));
                atomicMin(&out, o);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s.tile_left[t] = matches;
            atomicMin(L.first_out + tile.x, out);
        }
        __syncthreads();
    }
}

// The left sides, in order, and the positions they came from (T).
__global__ void __launch_bounds__(BB) k_sah_front(SahView s, uint32_t level) {
    __shared__ uint32_t before, all_left, chunk[SAH_TILE / 32];
    const SahLevel& L = s.level[level & 1];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tiles = s.ctl->failed ? 0u : s.ctl->tiles[level];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint2 tile = L.tiles[t];
        const SahNode& nd = L.nodes[tile.x];
        const uint32_t first = nd.first, count = nd.count, best = s.best[tile.x], p1 = L.first_out[tile.x];
        const uint32_t* src = s.order[level & 1];
        uint32_t* dst = s.order[(level & 1) ^ 1];
        if (threadIdx.x == 0) before = all_left = 0;
        __syncthreads();
        uint32_t mine = 0, total = 0;
        const uint32_t t0 = L.tile0[tile.x], nt = (count + SAH_TILE - 1) / SAH_TILE;
        for (uint32_t k = threadIdx.x; k < nt; k += BB) {
            const uint32_t v = s.tile_left[t0 + k];
            total += v;
            if (k < tile.y) mine += v;
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0) {
            atomicAdd(&before, mine);
            atomicAdd(&all_left, total);
        }
        unsigned left = 0;  // bit e: this thread's element e goes to the left
        for (uint32_t e = 0; e < SAH_TILE / BB; ++e) {
            const uint32_t i = tile.y * SAH_TILE + e * BB + threadIdx.x;
            const bool l = i < count && s.bucket[first + i] <= best;
            left |= l ? 1u << e : 0u;
            const unsigned m = __ballot_sync(0xffffffffu, l);
            if (lane == 0) chunk[e * SAH_WARPS + warp] = __popc(m);
        }
        __syncthreads();
        if (warp == 0) {  // exclusive scan of the 32 chunks
            const uint32_t c = chunk[lane];
            uint32_t x = c;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= static_cast<unsigned>(o)) x += y;
            }
            chunk[lane] = x - c;
        }
        __syncthreads();
        for (uint32_t e = 0; e < SAH_TILE / BB; ++e) {
            const uint32_t i = tile.y * SAH_TILE + e * BB + threadIdx.x;
            const bool l = (left >> e) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, l);
            if (!l) continue;
            const uint32_t rank = before + chunk[e * SAH_WARPS + warp] + __popc(m & ((1u << lane) - 1u));
            if (rank >= count) continue;
            dst[first + rank] = src[first + i];
            if (i > p1 && rank >= p1) s.moved[first + rank - p1] = i;
        }
        if (threadIdx.x == 0 && tile.y == 0) s.left[tile.x] = all_left;
        __syncthreads();
    }
}
static_assert(SAH_TILE / 32 == 32 && SAH_TILE % BB == 0, "a tile's chunks are one warp's scan");

// The right sides, and the children.
__global__ void __launch_bounds__(BB) k_sah_back(SahView s, uint32_t level) {
    const SahLevel& L = s.level[level & 1];
    // (one lane's reading: `failed` may be set by another block meanwhile)
    const uint32_t tiles = __shfl_sync(0xffffffffu, s.ctl->failed ? 0u : s.ctl->tiles[level], 0);
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint2 tile = L.tiles[t];
        const SahNode& nd = L.nodes[tile.x];
        const uint32_t first = nd.first, count = nd.count, best = s.best[tile.x], p1 = L.first_out[tile.x];
        const uint32_t k = s.left[tile.x], R = k - p1;
        const uint32_t* src = s.order[level & 1];
        uint32_t* dst = s.order[(level & 1) ^ 1];
        for (uint32_t e = 0; e < SAH_TILE; e += BB) {
            const uint32_t i = tile.y * SAH_TILE + e + threadIdx.x;
            if (i >= count || s.bucket[first + i] <= best) continue;
            const uint32_t to = first + k + sah_back(s.moved + first, i - p1, R, p1) - R;
            if (to < s.n) dst[to] = src[first + i];
        }
        if (tile.y != 0 || threadIdx.x >= 64) continue;
        // The children: a warp each.
        const uint32_t side = threadIdx.x >> 5, id = first + k - 1;
        const int* tab = L.tables + tile.x * (SAH_BUCKETS * SAH_VALUES);
        SahNode c;
        c.first = side ? first + k : first;
        c.count = side ? count - k : k;
        c.slot = 2 * id + side;
        c.range = nd.range;
        for (int a = 0; a < 3; ++a) {
            c.box[a] = c.cb[a] = FLT_MAX;
            c.box[3 + a] = c.cb[3 + a] = -FLT_MAX;
        }
        const uint32_t from = side ? best + 1 : 0, to = side ? SAH_BUCKETS : best + 1;
        for (uint32_t b = from; b < to; ++b)
            for (int a = 0; a < 3; ++a) {
                const int* v = tab + b * SAH_VALUES;
                c.box[a] = fminf(c.box[a], unordered(v[1 + a]));
                c.box[3 + a] = fmaxf(c.box[3 + a], unordered(v[4 + a]));
                c.cb[a] = fminf(c.cb[a], unordered(v[7 + a]));
                c.cb[3 + a] = fmaxf(c.cb[3 + a], unordered(v[10 + a]));
            }
        if (k == 0 || k >= count) {  // cannot be: the first and last buckets hold components
            if (threadIdx.x == 0) atomicExch(&s.ctl->failed, 1u);
            continue;
        }
        if ((threadIdx.x & 31u) == 0 && GR_IN_RANGE(c.slot, 2 * (s.n - 1))) {
            float* o = s.opened + 8 * static_cast<size_t>(c.slot);
            for (int a = 0; a < 3; ++a) {
                o[a] = c.box[a];
                o[4 + a] = c.box[3 + a];
            }
            o[7] = __int_as_float(static_cast<int>(c.count));
            if (side == 0) {
                if (nd.slot == SAH_ROOT) s.ctl->root = static_cast<int>(id);
                else s.opened[8 * static_cast<size_t>(nd.slot) + 3] = __int_as_float(static_cast<int>(id));
            }
        }
        sah_enter(s, level + 1, c);
    }
}

// A subtree in shared memory, of at most N components.
template <uint32_t N>
struct SahTree {
    float box[6][N];
    uint32_t id[N];
    uint16_t order[2][N], moved[N];
    uint8_t bucket[N];
    int tab[SAH_WARPS][SAH_BUCKETS * SAH_VALUES];
    uint2 list[2][N / 4];  // nodes of more than four: (first | count << 16, slot | range << 31)
    uint2 tiny[N / 2];     // nodes of two to four
    uint32_t listed[2], tinies;
    GR_D float cen(uint32_t k, int dim) const {
        k %= N;
        return 0.5f * box[dim][k] + 0.5f * box[3 + dim][k];
    }
};
static_assert(sizeof(SahTree<SAH_SMALL_MANY>) <= 48 * 1024, "k_sah_small is launched without a shared memory attribute");
constexpr uint32_t SAH_RANGE = 1u << 31;

// The reference's nth_element (geom/util.rs), its swap partition and its shortened left side
// included, on `s`.
template <uint32_t N>
GR_D void sah_nth(const SahTree<N>& T, uint16_t* s, uint32_t len, uint32_t nth, int dim) {
    while (len >= 2) {
        const uint32_t pivot = len / 2;
        const uint16_t pe = s[pivot];
        s[pivot] = s[len - 1];
        s[len - 1] = pe;
        const float pv = T.cen(pe, dim);
        uint32_t at = 0;
        for (uint32_t i = 0; i + 1 < len; ++i) {
            const uint16_t e = s[i];
            if (T.cen(e, dim) < pv) {
                s[i] = s[at];
                s[at++] = e;
            }
        }
        s[len - 1] = s[at];
        s[at] = pe;
        if (nth < at) {
            len = at - 1;
        } else if (nth > at) {
            s += at + 1;
            len -= at + 1;
            nth -= at + 1;
        } else {
            return;
        }
    }
}

GR_D void sah_slot(const SahView& s, uint32_t slot, const float* b, int ref, uint32_t count) {
    if (!GR_IN_RANGE(slot, 2 * (s.n - 1))) return;
    float4* o = reinterpret_cast<float4*>(s.opened + 8 * static_cast<size_t>(slot));
    o[0] = make_float4(b[0], b[1], b[2], __int_as_float(ref));
    o[1] = make_float4(b[3], b[4], b[5], __int_as_float(static_cast<int>(count)));
}

// A single component at position `at` of the subtree: its slot and its place in the order.
template <uint32_t N>
GR_D void sah_single(const SahView& s, const SahTree<N>& T, uint32_t first, uint32_t at, uint32_t e, uint32_t slot,
                     uint32_t* __restrict__ perm) {
    float b[6];
    e %= N;
    for (int a = 0; a < 6; ++a) b[a] = T.box[a][e];
    sah_slot(s, slot, b, ~static_cast<int>(first + at), 1);
    if (GR_IN_RANGE(first + at, s.n)) perm[first + at] = T.id[e];
}

// Subtrees of two to four components, by one thread.
template <uint32_t N>
GR_D void sah_tiny(const SahView& s, SahTree<N>& T, uint32_t first, uint16_t* order, uint2 node, uint32_t* perm) {
    uint2 todo[4];
    int left = 0;
    todo[left++] = node;
    while (left) {
        const uint2 nd = todo[--left];
        const uint32_t f = nd.x & 0xFFFFu, n = nd.x >> 16, slot = nd.y & ~SAH_RANGE;
        if (n == 1) {
            sah_single(s, T, first, f, order[f], slot, perm);
            continue;
        }
        float b[6], cb[6];
        for (int a = 0; a < 3; ++a) {
            b[a] = cb[a] = FLT_MAX;
            b[3 + a] = cb[3 + a] = -FLT_MAX;
        }
        for (uint32_t i = f; i < f + n; ++i) {
            const uint32_t e = order[i] % N;
            for (int a = 0; a < 3; ++a) {
                const float c = T.cen(e, a);
                b[a] = fminf(b[a], T.box[a][e]);
                b[3 + a] = fmaxf(b[3 + a], T.box[3 + a][e]);
                cb[a] = fminf(cb[a], c);
                cb[3 + a] = fmaxf(cb[3 + a], c);
            }
        }
        uint32_t range = nd.y & SAH_RANGE;
        const int dim = max_extent6(cb);
        if (!range && cb[dim] == cb[3 + dim]) {
            range = SAH_RANGE;
            atomicAdd(&s.ctl->excess, n - 1);
        }
        const uint32_t mid = n / 2, id = first + f + mid - 1;
        if (!range) sah_nth(T, order + f, n, mid, dim);
        sah_slot(s, slot, b, static_cast<int>(id), n);
        todo[left++] = make_uint2((f + mid) | ((n - mid) << 16), (2 * id + 1) | range);
        todo[left++] = make_uint2(f | (mid << 16), (2 * id) | range);
    }
}

// Builds the small subtrees, a block each, level by level: a warp a node, then a thread per
// node of at most four components.  Bound by the chain of a warp's reductions in the first
// levels and by the serial nth_element of the last ones.
template <uint32_t N>
__global__ void __launch_bounds__(BB) k_sah_small(SahView s, uint32_t* __restrict__ perm) {
    extern __shared__ unsigned char smem[];
    SahTree<N>& T = *reinterpret_cast<SahTree<N>*>(smem);
    const unsigned all = 0xffffffffu, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    // (not launched once `failed` is set; a block that sets it below has a tree all the same, and
    // the barriers need every thread of a block to make the same turns)
    const uint32_t trees = s.ctl->small;
    int* tab = T.tab[warp];
    for (uint32_t t = blockIdx.x; t < trees; t += gridDim.x) {
        const SahSmall root = s.small[t];
        const uint32_t first = root.first;
        for (uint32_t k = threadIdx.x; k < root.count; k += BB) {
            const uint32_t id = s.order[root.flags >> 1][first + k];
            float x[6], c[3];
            sah_load(s, id, x, c);
            for (int a = 0; a < 6; ++a) T.box[a][k] = x[a];
            T.id[k] = id;
            T.order[0][k] = static_cast<uint16_t>(k);
        }
        if (threadIdx.x == 0) {
            const uint2 nd = make_uint2(root.count << 16, root.slot | (root.flags & 1u ? SAH_RANGE : 0u));
            T.listed[0] = T.listed[1] = T.tinies = 0;
            if (root.count > 4) T.list[0][T.listed[0]++] = nd;
            else T.tiny[T.tinies++] = nd;
        }
        __syncthreads();
        // A level leaves every node smaller: it ends.
        for (uint32_t depth = 0; depth <= N; ++depth) {
            const int cur = depth & 1;
            uint16_t *A = T.order[cur], *B = T.order[cur ^ 1];
            const uint32_t nodes = T.listed[cur];
            for (uint32_t w = warp; w < nodes; w += SAH_WARPS) {
                const uint2 nd = T.list[cur][w];
                const uint32_t f = nd.x & 0xFFFFu, n = nd.x >> 16;
                uint32_t range = nd.y & SAH_RANGE;
                int v[12];  // ordered bounds: box lo, hi, centroid lo, hi
                for (int a = 0; a < 12; ++a) v[a] = a / 3 % 2 ? static_cast<int>(0x80000000u) : 0x7FFFFFFF;
                for (uint32_t j = lane; j < n; j += 32) {
                    const uint32_t e = A[f + j] % N;
                    for (int a = 0; a < 3; ++a) {
                        const int c = ordered(T.cen(e, a));
                        v[a] = min(v[a], ordered(T.box[a][e]));
                        v[3 + a] = max(v[3 + a], ordered(T.box[3 + a][e]));
                        v[6 + a] = min(v[6 + a], c);
                        v[9 + a] = max(v[9 + a], c);
                    }
                }
                float b[6], cb[6];
                for (int a = 0; a < 6; ++a) {
                    b[a] = unordered(a < 3 ? __reduce_min_sync(all, v[a]) : __reduce_max_sync(all, v[a]));
                    cb[a] = unordered(a < 3 ? __reduce_min_sync(all, v[6 + a]) : __reduce_max_sync(all, v[6 + a]));
                }
                const int dim = max_extent6(cb);
                const float lo = dim == 0 ? cb[0] : (dim == 1 ? cb[1] : cb[2]);
                const float hi = dim == 0 ? cb[3] : (dim == 1 ? cb[4] : cb[5]);
                if (!range && lo == hi) {
                    range = SAH_RANGE;
                    if (lane == 0) atomicAdd(&s.ctl->excess, n - 1);
                }
                uint32_t mid = n / 2;
                bool sorted = range != 0;  // the order stands, in A
                if (!range) {
                    for (uint32_t k = lane; k < SAH_BUCKETS * SAH_VALUES; k += 32)
                        tab[k] = sah_empty(static_cast<int>(k % SAH_VALUES));
                    __syncwarp();
                    for (uint32_t j0 = 0; j0 < n; j0 += 32) {
                        const uint32_t j = j0 + lane;
                        const bool in = j < n;
                        float x[6] = {}, c[3] = {};
                        uint32_t k = 0;
                        if (in) {
                            const uint32_t e = A[f + j] % N;
                            for (int a = 0; a < 6; ++a) x[a] = T.box[a][e];
                            for (int a = 0; a < 3; ++a) c[a] = 0.5f * x[a] + 0.5f * x[3 + a];
                            k = sah_bucket(dim == 0 ? c[0] : (dim == 1 ? c[1] : c[2]), lo, hi);
                            T.bucket[f + j] = static_cast<uint8_t>(k);
                        }
                        sah_add<false>(tab, in, k, x, c);
                    }
                    float cost;
                    const uint32_t best = sah_best(tab, b, cost);
                    if (n > 255 || cost < static_cast<float>(n)) {
                        // The swap partition, as in k_sah_front and k_sah_back.
                        uint32_t k = 0, p1 = n;
                        for (uint32_t j0 = 0; j0 < n; j0 += 32) {
                            const bool in = j0 + lane < n, l = in && T.bucket[f + j0 + lane] <= best;
                            const unsigned m = __ballot_sync(all, l), o = __ballot_sync(all, in && !l);
                            if (o && p1 == n) p1 = j0 + __ffs(o) - 1;
                            k += __popc(m);
                        }
                        const uint32_t R = k - p1;
                        uint32_t rank = 0;
                        for (uint32_t j0 = 0; j0 < n; j0 += 32) {
                            const uint32_t j = j0 + lane;
                            const bool l = j < n && T.bucket[f + j] <= best;
                            const unsigned m = __ballot_sync(all, l);
                            if (l) {
                                const uint32_t q = rank + __popc(m & below);
                                B[f + q] = A[f + j];
                                if (j > p1) T.moved[f + q - p1] = static_cast<uint16_t>(j);
                            }
                            rank += __popc(m);
                        }
                        __syncwarp();
                        for (uint32_t j = lane; j < n; j += 32) {
                            if (T.bucket[f + j] <= best) continue;
                            const uint32_t to = f + k + sah_back(T.moved + f, j - p1, R, p1) - R;
                            if (to < N) B[to] = A[f + j];
                        }
                        mid = k;
                        if (k == 0 || k >= n) {  // cannot be: the first and last buckets hold components
                            if (lane == 0) atomicExch(&s.ctl->failed, 1u);
                            mid = n / 2;
                            sorted = true;
                        }
                    } else {
                        __syncwarp();
                        if (lane == 0) sah_nth(T, A + f, n, mid, dim);
                        sorted = true;
                    }
                }
                __syncwarp();
                if (sorted)
                    for (uint32_t j = lane; j < n; j += 32) B[f + j] = A[f + j];
                __syncwarp();
                const uint32_t id = first + f + mid - 1;
                if (lane == 0) sah_slot(s, nd.y & ~SAH_RANGE, b, static_cast<int>(id), n);
                if (lane < 2) {
                    const uint32_t cf = lane ? f + mid : f, cn = lane ? n - mid : mid, slot = 2 * id + lane;
                    const uint2 c = make_uint2(cf | (cn << 16), slot | range);
                    if (cn > 4) {
                        const uint32_t at = atomicAdd(&T.listed[cur ^ 1], 1u);
                        if (GR_IN_RANGE(at, N / 4)) T.list[cur ^ 1][at] = c;
                    } else if (cn > 1) {
                        const uint32_t at = atomicAdd(&T.tinies, 1u);
                        if (GR_IN_RANGE(at, N / 2)) T.tiny[at] = c;
                    } else sah_single(s, T, first, cf, B[cf], slot, perm);
                }
            }
            __syncthreads();
            // (the first level's nodes of at most four are in A)
            uint16_t* at = depth == 0 && root.count <= 4 ? A : B;
            for (uint32_t w = threadIdx.x; w < T.tinies; w += BB) sah_tiny(s, T, first, at, T.tiny[w], perm);
            __syncthreads();
            const bool end = T.listed[cur ^ 1] == 0;
            __syncthreads();
            if (threadIdx.x == 0) T.listed[cur] = T.tinies = 0;
            if (end) break;
            __syncthreads();
        }
        __syncthreads();
    }
}

}  // namespace

}  // namespace gr
