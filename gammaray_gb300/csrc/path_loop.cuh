// The path loop: few paths carried to their end in one launch, shared by the path tracer,
// BDPT's walks and the batch engine.
#pragma once

#include "traverse.cuh"

namespace gr {

// Queues of at most PATH_LOOP_MAX paths are carried to their end by one launch
// (k_pt_finish) instead of an extension and a shading launch per bounce; a group that
// starts that small needs no queue at all.  Below it a bounce is bounded by latency: its
// two launches take about 30 us however few paths are left, and on meshes the slowest ray
// of each bounce alone takes 90-140 us.  Above it the wavefront's sorted shading and
// refilled extension win.  Measured, wavefront against path loop (us per render):
//   Cornell box, depth 8     5 k paths 377 / 181, 66 k 400 / 258, 393 k 545 / 611
//   50 k triangles, depth 12 8 k paths - / 295, 240 k 1361 / 598, 393 k 955 / 760
//   102 k triangles, 66 k paths 1256 / 463
// and as the end of a larger render: 641 x 359 x 9 spp, unbounded depth 2439 -> 1695,
// 512 x 512 x 4 spp 2080 -> 1480, 1024 x 1024 x 64 spp 28.61 -> 28.40 ms.  Taking over at
// 2^18 / 2^19 / 2^20 paths: 1242 / 1330 / 1308 us on the second of these, 1.10 / 1.22 / 1.42
// ms on 1 M paths of the Cornell box.
constexpr uint32_t PATH_LOOP_MAX = 1u << 18;
// Depths the path loop takes: one launch carries a path to its end, so its length has to
// be bounded, by max_depth or by the roulette (at most 3/4 survive a bounce beyond
// rr_aggressive_depth).  Other settings keep a launch per bounce.
constexpr uint32_t PATH_LOOP_DEPTH = 256;
constexpr uint32_t PATH_LOOP_RR_DEPTH = 64;
// At 4 blocks per SM it has 128 registers; it uses 112.
constexpr int PATH_LOOP_BLOCKS = 4;
// Lanes of a warp that carry paths when there are too few to fill every warp: lanes of a
// warp wait for each other, but fewer lanes per warp repeat the shading code.  4 / 8 / 16
// / 32 measured 193 / 181 / 170 / 181 us on 5 k paths of the Cornell box, 280 / 295 / 316
// / 324 us on 8 k of a mesh.
constexpr uint32_t PATH_LOOP_MIN_LANES = 8;

// Path loop: a warp carries paths from their first ray to their end without going back
// to a queue.  Its lanes trace, one traversal step each per iteration, until every path
// of the warp has its closest hit, then all of them shade, and the survivors trace their
// next rays; lanes whose paths ended take other paths.  One launch replaces an extension
// and a shading launch per bounce, and a slow ray delays its own warp's paths instead of
// every path of its bounce.
//   n       paths; path index q goes to take() once
//   fetch   a zeroed counter; the first paths, one per lane, are handed out by position
//           (neighbouring ones to different blocks, so a costly part of an image does not
//           fall on one SM), the rest from it
//   scene()               this lane's scene: nodes, prims and step budget
//   take(q, o, d)         loads path q and its next ray; false: it has none
//   shade(q, t, no, nd)   shades the hit in t (t.hit, t.closest, t.hu, t.hv); true and the
//                         next ray in (no, nd) when the path goes on
// Every warp intrinsic runs where control flow is warp-uniform (each condition around one
// comes from ballots or from the shuffled base), and every loop ends: a traversal
// iteration steps a lane whose ray has the scene's step budget, each path is handed out
// once and ends by its depth limit or roulette.  Returns the rays this lane traced.
template <int W, class K, class SceneOf, class Take, class Shade>
GR_D uint32_t run_paths(const K& stk, uint32_t n, uint32_t* fetch, int* err, int* err_ray, const SceneOf& scene,
                        const Take& take, const Shade& shade) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    // Lanes of a warp that carry paths: as many as spread them over the whole grid, since
    // lanes of one warp wait for each other.
    const uint32_t lanes = min(32u, max(PATH_LOOP_MIN_LANES, (n + warps - 1) / warps));
    const bool use = lane < lanes;
    const uint32_t first = warps * lanes;  // paths handed out by position
    const uint32_t refill_at = lanes < 4u ? 1u : lanes / 4u;
    TravState t;
    t.hit = -1;
    uint32_t q = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * lanes + lane, steps = 0, traced = 0;
    bool busy = false, exhausted = first >= n;
    auto start = [&](V3 o, V3 d) {
        trav_init(t, o, d, FLT_MAX);
        steps = 0;
        ++traced;
        busy = true;
    };
    if (use && q < n) {
        V3 o, d;
        if (take(q, o, d)) start(o, d);
    }
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, use && !busy);
        if (!exhausted && static_cast<uint32_t>(__popc(idle)) >= refill_at) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(fetch, static_cast<uint32_t>(__popc(idle)));
            base = __shfl_sync(0xffffffffu, base, 0) + first;
            exhausted = static_cast<uint64_t>(base) + __popc(idle) >= n;
            if (use && !busy) {
                q = base + __popc(idle & below);
                V3 o, d;
                if (q < n && take(q, o, d)) start(o, d);
            }
        }
        // No lane busy and paths left: every lane is idle, so the next iteration takes
        // paths or learns that none are left.
        if (__ballot_sync(0xffffffffu, busy) == 0u && exhausted) break;
        bool trav = busy;
        while (__any_sync(0xffffffffu, trav)) {
            if (trav) {
                bool done = trav_step<W, false, false>(scene(), t, stk, err, nullptr);
                if (!done && ++steps > scene().step_budget) {
                    atomicExch(err, 2);
                    if (err_ray) atomicExch(err_ray, static_cast<int>(q));
                    t.hit = -1;
                    done = true;
                }
                trav = !done;
            }
        }
        if (busy) {
            V3 no, nd;
            if (shade(q, t, no, nd)) start(no, nd);
            else busy = false;
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
