// The path loop: few paths carried to their end in one launch, shared by the path tracer,
// BDPT's walks and the batch engine.
#pragma once

#include "shade_sort.cuh"
#include "traverse.cuh"

namespace gr {

// Queues of at most PATH_LOOP_MAX paths are carried to their end by one launch
// (k_pt_finish) instead of an extension and a shading launch per bounce; a group that
// starts that small needs no queue at all.  Below it a bounce is bounded by latency: its
// two launches take about 30 us however few paths are left, and on meshes the slowest ray
// of each bounce alone takes 90-140 us.  Above it the wavefront's refilled extension wins.
// Measured, wavefront against path loop (us per render):
//   Cornell box, depth 8     5 k paths 377 / 157, 66 k 400 / 220
//   50 k triangles, depth 12 240 k paths 1361 / 486
// and as the end of a larger render: 641 x 359 x 9 spp, unbounded depth 2439 -> 1388,
// 512 x 512 x 4 spp 2080 -> 1181.  Taking over at 2^17 / 2^18 / 2^19 paths: 1404 / 1388 /
// 1395 us and 1253 / 1181 / 1167 on these two, 618 / 487 / 487 on 240 k paths of 50 k
// triangles, 1054 / 1094 / 1146 on 1 M paths of the Cornell box, 1258 / 1202 / 1239 on BDPT
// of a mesh (300 x 300 x 4 spp).
constexpr uint32_t PATH_LOOP_MAX = 1u << 18;
// Depths the path loop takes: one launch carries a path to its end, so its length has to
// be bounded, by max_depth or by the roulette (at most 3/4 survive a bounce beyond
// rr_aggressive_depth).  Other settings keep a launch per bounce.
constexpr uint32_t PATH_LOOP_DEPTH = 256;
constexpr uint32_t PATH_LOOP_RR_DEPTH = 64;
// Threads of a block, which shades its paths together (run_paths), and blocks per SM: 128
// registers.  A warp shading its own 13 paths or so (of 32 lanes, the others waiting for
// paths to end) ran 50,000 cycles for it, since its lanes take different lobes and the code
// of all of them passes through the instruction cache; sorted over 256 threads 8,000.
// Blocks of 64 / 128 / 256 / 512 threads: 1,519 / 1,437 / 1,386 / 1,397 us for 641 x 359 x 9
// spp of a mesh, 904 / 865 / 812 / 786 for BDPT of the Cornell box (200 x 150 x 4 spp), 169 /
// 157 / 157 / 169 for 96 x 54 paths of it; warp by warp 1,480, 822 and 167.
constexpr int PATH_LOOP_THREADS = 256;
constexpr int PATH_LOOP_BLOCKS = 2;
// Lanes of a warp that carry paths when there are too few to fill every warp: lanes of a
// warp wait for each other.  4 / 8 measured 157 / 157 us for 96 x 54 paths of the Cornell
// box, 487 / 486 for 300 x 200 x 4 spp of a mesh.
constexpr uint32_t PATH_LOOP_MIN_LANES = 8;
// A block's shared memory: its threads' traversal stacks, their paths (word by word, a
// column each), and the shading order.
constexpr size_t path_loop_smem_bytes(int words) {
    return step_stack_smem_bytes(PATH_LOOP_THREADS) +
           static_cast<size_t>(words + 1) * sizeof(uint32_t) * PATH_LOOP_THREADS +
           (SORT_BUCKETS + 1) * sizeof(uint32_t);
}

// Path loop: a block carries paths from their first ray to their end without going back to
// a queue.  Its lanes trace, one traversal step each per iteration, until every path of the
// block has its closest hit; the block sorts the hits by code path (shade_bucket), and its
// warps shade them in that order, each an equal share.
// One launch replaces an extension and a shading launch per bounce, and a slow ray delays
// its own block's paths instead of every path of its bounce.
//   n       paths; path index q goes to take() once
//   fetch   a zeroed counter; the first paths, one per lane, are handed out by position
//           (neighbouring ones to different blocks, so a costly part of an image does not
//           fall on one SM), the rest from it
//   grouped               trace a warp's last rays by groups of lanes
//   scene()               this lane's scene: nodes, prims and step budget
//   take(q, path, o, d)   loads path q and its next ray
//   bucket(path, k)       shading bucket and lobe (shade_bucket) of its hit k
//   shade(path, lobe, o, d, h, no, nd)   shades the hit h = (t, k, u, v) of the ray (o, d);
//                         true and the next ray when the path goes on
// P is moved between threads word by word, its first WORDS words.
// Every barrier and warp intrinsic runs where control flow is uniform (each condition around
// one comes from the block's count, from ballots or from a shuffled base), and every loop
// ends: a traversal iteration steps a lane whose ray has the scene's step budget, each path
// is handed out once and ends by its depth limit or roulette.  A warp without a path has
// learned that none are left, so the block ends when no lane has one.  Returns the rays
// this lane traced.
template <int W, int WORDS, class P, class K, class SceneOf, class Take, class Bucket, class Shade>
GR_D uint32_t run_paths(const K& stk, unsigned char* smem, uint32_t n, uint32_t* fetch, int* err, int* err_ray,
                        bool grouped, const SceneOf& scene, const Take& take, const Bucket& bucket,
                        const Shade& shade) {
    constexpr int NT = PATH_LOOP_THREADS;
    static_assert(sizeof(P) % 4 == 0 && WORDS * 4 <= sizeof(P), "whole words");
    static_assert(SMEM_STACK >= 5, "a ray and its hit in a finished stack's column");
    uint32_t* paths = reinterpret_cast<uint32_t*>(smem + step_stack_smem_bytes(NT));
    uint32_t* order = paths + WORDS * NT;
    uint32_t* count = order + NT;
    uint32_t* total = count + SORT_BUCKETS;
    int2* rays = reinterpret_cast<int2*>(smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t warps = gridDim.x * (NT / 32);
    auto load_path = [&](uint32_t at, P& p) {
        uint32_t w[sizeof(P) / 4] = {};
#pragma unroll
        for (int k = 0; k < WORDS; ++k) w[k] = paths[k * NT + at];
        memcpy(&p, w, sizeof(P));
    };
    auto store_path = [&](uint32_t at, const P& p) {
        uint32_t w[sizeof(P) / 4];
        memcpy(w, &p, sizeof(P));
#pragma unroll
        for (int k = 0; k < WORDS; ++k) paths[k * NT + at] = w[k];
    };
    // Lanes of a warp that carry paths: as many as spread them over the whole grid, since
    // lanes of one warp wait for each other.
    const uint32_t lanes = min(32u, max(PATH_LOOP_MIN_LANES, (n + warps - 1) / warps));
    const bool use = lane < lanes;
    const uint32_t first = warps * lanes;  // paths handed out by position
    const uint32_t refill_at = lanes < 4u ? 1u : lanes / 4u;
    TravState t;
    t.hit = -1;
    uint32_t q = ((tid >> 5) * gridDim.x + blockIdx.x) * lanes + lane, steps = 0, traced = 0;
    bool busy = false, exhausted = first >= n;
    auto start = [&](V3 o, V3 d) {
        trav_init(t, o, d, FLT_MAX);
        steps = 0;
        ++traced;
        busy = true;
    };
    auto begin = [&]() {
        P p;
        V3 o, d;
        take(q, p, o, d);
        store_path(tid, p);
        start(o, d);
    };
    if (tid < SORT_BUCKETS) count[tid] = 0;
    if (use && q < n) begin();
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, use && !busy);
        if (!exhausted && static_cast<uint32_t>(__popc(idle)) >= refill_at) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(fetch, static_cast<uint32_t>(__popc(idle)));
            base = __shfl_sync(0xffffffffu, base, 0) + first;
            exhausted = static_cast<uint64_t>(base) + __popc(idle) >= n;
            if (use && !busy) {
                q = base + __popc(idle & below);
                if (q < n) begin();
            }
        }
        if (!__syncthreads_or(busy)) break;
        bool trav = busy, deep = false;  // deep: grouped lanes gave this ray back
        for (;;) {
            const unsigned left = __ballot_sync(0xffffffffu, trav);
            if (left == 0u) break;
            const unsigned last = grouped ? __ballot_sync(0xffffffffu, trav && !deep) : 0u;
            bool over = false;
            if (last && __popc(last) <= 32 / W) {
                trace_grouped<W, false>(last, scene(), t, steps, stk, deep, over);
                trav = trav && deep;
            } else if (trav) {
                const bool done = trav_step<W>(scene(), t, stk, err);
                over = !done && ++steps > scene().step_budget;
                trav = !done && !over;
            }
            if (over) {
                atomicExch(err, 2);
                if (err_ray) atomicExch(err_ray, static_cast<int>(q));
                t.hit = -1;
            }
        }
        uint32_t b = 0, pos = 0;
        if (busy) {
            rays[tid] = make_int2(__float_as_int(t.o.x), __float_as_int(t.o.y));
            rays[NT + tid] = make_int2(__float_as_int(t.o.z), __float_as_int(t.d.x));
            rays[2 * NT + tid] = make_int2(__float_as_int(t.d.y), __float_as_int(t.d.z));
            rays[3 * NT + tid] = make_int2(__float_as_int(t.closest), t.hit);
            rays[4 * NT + tid] = make_int2(__float_as_int(t.hu), __float_as_int(t.hv));
            P p;
            load_path(tid, p);
            b = bucket(p, t.hit);
            pos = atomicAdd(count + b % SORT_BUCKETS, 1u);
        }
        __syncthreads();
        if (tid < 32) {  // exclusive scan of the bucket sizes
            const uint32_t c = count[tid];
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= static_cast<uint32_t>(o)) x += y;
            }
            count[tid] = x - c;
            if (tid == 31) *total = x;
        }
        __syncthreads();
        if (busy && GR_IN_RANGE(count[b % SORT_BUCKETS] + pos, NT))
            order[count[b % SORT_BUCKETS] + pos] = tid | (b / SORT_BUCKETS << 16);
        __syncthreads();
        const uint32_t m = *total, share = (m + NT / 32 - 1) / (NT / 32), at = (tid >> 5) * share + lane;
        if (tid < SORT_BUCKETS) count[tid] = 0;
        if (lane < share && at < m) {
            const uint32_t from = order[at] & 0xFFFFu, lobe = order[at] >> 16;
            const int2 r0 = rays[from], r1 = rays[NT + from], r2 = rays[2 * NT + from], r3 = rays[3 * NT + from],
                       r4 = rays[4 * NT + from];
            P p;
            load_path(from, p);
            V3 no, nd;
            const float4 h = make_float4(__int_as_float(r3.x), __int_as_float(r3.y), __int_as_float(r4.x),
                                         __int_as_float(r4.y));
            const bool alive = shade(p, lobe, V3{__int_as_float(r0.x), __int_as_float(r0.y), __int_as_float(r1.x)},
                                     V3{__int_as_float(r1.y), __int_as_float(r2.x), __int_as_float(r2.y)}, h, no, nd);
            rays[3 * NT + from] = make_int2(alive ? 1 : 0, 0);
            if (alive) {
                store_path(from, p);
                rays[from] = make_int2(__float_as_int(no.x), __float_as_int(no.y));
                rays[NT + from] = make_int2(__float_as_int(no.z), __float_as_int(nd.x));
                rays[2 * NT + from] = make_int2(__float_as_int(nd.y), __float_as_int(nd.z));
            }
        }
        __syncthreads();
        if (busy) {
            busy = rays[3 * NT + tid].x != 0;
            if (busy) {
                const int2 r0 = rays[tid], r1 = rays[NT + tid], r2 = rays[2 * NT + tid];
                start(V3{__int_as_float(r0.x), __int_as_float(r0.y), __int_as_float(r1.x)},
                      V3{__int_as_float(r1.y), __int_as_float(r2.x), __int_as_float(r2.y)});
            }
        }
    }
    return traced;
}

// Adds the warp's traced rays to *rays (one atomic per warp; every lane calls it).
GR_D void count_rays(uint32_t traced, unsigned long long* rays) {
    const uint32_t sum = __reduce_add_sync(0xffffffffu, traced);
    if ((threadIdx.x & 31u) == 0 && sum) atomicAdd(rays, static_cast<unsigned long long>(sum));
}

// Whether one launch can carry paths with these limits to their end.
inline bool path_loop_bounded(uint32_t max_depth, uint32_t rr_depth, uint32_t rr_aggressive_depth) {
    if (max_depth) return max_depth <= PATH_LOOP_DEPTH;
    return rr_depth <= PATH_LOOP_RR_DEPTH && rr_aggressive_depth <= PATH_LOOP_RR_DEPTH;
}

}  // namespace gr
