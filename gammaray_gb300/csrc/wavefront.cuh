// Pieces shared by the wavefront integrators (pt.cu, bdpt.cu): the extension kernel
// over a compacted ray queue, the warp-aggregated queue push and grid sizing.
#pragma once

#include <algorithm>
#include <cstdlib>

#include "runtime.hpp"
#include "shade_sort.cuh"
#include "traverse.cuh"


namespace gr {
namespace {

constexpr int BLOCK = 128;

// Shading kernels are register-heavy (the Disney mixture); asking for 6 resident blocks
// of 128 threads caps them at 85 registers, which measured 3% faster on the bench
// workload than the uncapped 96 (occupancy 31% -> 37%).  GR_SHADE_MIN_BLOCKS overrides.
#ifndef GR_SHADE_MIN_BLOCKS
#define GR_SHADE_MIN_BLOCKS 6
#endif
#define GR_SHADE_BOUNDS __launch_bounds__(BLOCK, GR_SHADE_MIN_BLOCKS)

// Closest hit for every queued ray (trace_queue); the queue's length is read on the
// device, so launches never depend on a host read of it.
// one_origin: every ray of the queue starts at q_o[0] (the path tracer's camera rays:
// one pinhole origin, stored once).
// At 54 registers 9 blocks fit an SM; capped for 10 (some spilled) the extension of the
// path-tracer workload took 15.5 instead of 14.0 ms per render.
template <int W, bool COUNT>
__global__ void __launch_bounds__(BLOCK) k_extend_refill(DeviceScene s, const uint32_t* __restrict__ count,
                                                  const float4* __restrict__ q_o, const float4* __restrict__ q_d,
                                                  float4* __restrict__ q_hit, int* err, unsigned long long* rays,
                                                  uint32_t* fetch, bool one_origin) {
    extern __shared__ unsigned char smem[];
    int2 spill[MAX_STACK - SMEM_STACK];
    const auto stk = thread_stack<BLOCK>(smem, spill);
    const uint32_t n = *count;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(rays, static_cast<unsigned long long>(n));
    uint32_t counts[2] = {0, 0};
    trace_queue<W, false, COUNT>(
        n, stk, err, err + 1, counts, SharedCounter{fetch}, [&]() -> const DeviceScene& { return s; },
        [&](uint32_t q, TravState& t) {
            const float4 o4 = q_o[one_origin ? 0u : q], d4 = q_d[q];
            trav_init(t, V3{o4.x, o4.y, o4.z}, V3{d4.x, d4.y, d4.z}, FLT_MAX);
            return true;
        },
        [&](uint32_t q, const TravState& t) {
            q_hit[q] = make_float4(t.closest, __int_as_float(t.hit), t.hu, t.hv);
        });
    if (COUNT && (counts[0] | counts[1])) {
        atomicAdd(rays + (CNT_NODES - CNT_RAYS) / 2, static_cast<unsigned long long>(counts[0]));
        atomicAdd(rays + (CNT_PRIMS - CNT_RAYS) / 2, static_cast<unsigned long long>(counts[1]));
    }
}

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
//   take(q, o, d)         loads path q and its next ray; false: it has none
//   shade(q, t, no, nd)   shades the hit in t (t.hit, t.closest, t.hu, t.hv); true and the
//                         next ray in (no, nd) when the path goes on
// Every warp intrinsic runs where control flow is warp-uniform (each condition around one
// comes from ballots or from the shuffled base), and every loop ends: a traversal
// iteration steps a lane whose ray has the scene's step budget, each path is handed out
// once and ends by its depth limit or roulette.  Returns the rays this lane traced.
template <int W, class K, class Take, class Shade>
GR_D uint32_t run_paths(const DeviceScene& s, const K& stk, uint32_t n, uint32_t* fetch, int* err, const Take& take,
                        const Shade& shade) {
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
                bool done = trav_step<W, false, false>(s, t, stk, err, nullptr);
                if (!done && ++steps > s.step_budget) {
                    atomicExch(err, 2);
                    atomicExch(err + 1, static_cast<int>(q));
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

// Blocks of `block` threads for n items: every block the device can hold at once (SMs x
// resident blocks per SM, asked of the current device at each launch), or fewer when n
// needs fewer.
template <class K>
int resident_grid(K kernel, size_t smem, uint32_t n, int block = BLOCK) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const int sm = device_sm_count();
    uint32_t need = (n + block - 1) / block;
    uint32_t cap = static_cast<uint32_t>(sm * per_sm);
    return static_cast<int>(std::max(1u, std::min(need, cap)));
}

// Grid of a path-loop kernel (blocks of BLOCK threads) for at most `most` paths.
template <class K>
int path_loop_grid(K kernel, size_t smem, uint32_t most) {
    return resident_grid(kernel, smem, (most + PATH_LOOP_MIN_LANES - 1) / PATH_LOOP_MIN_LANES * 32u);
}

// The start of a bounce whose queue is `cur`: a queue of at most `take` paths goes to the
// path loop (its length to CNT_LOOP, and the bounce's own launches find it empty).  The
// device decides, so the queue goes there at the first bounce that is short enough; the
// host reads (paths the loop takes, queue length) from `seen`, pinned host memory, while the
// bounce runs.  Clears the counters of the bounce's launches.
__global__ void k_bounce_begin(uint32_t* cnt, int cur, uint32_t take, uint32_t* seen) {
    const uint32_t q = cnt[cur];
    const bool taken = q <= take;
    cnt[CNT_LOOP] = taken ? q : 0u;
    if (taken) cnt[cur] = 0u;
    cnt[cur ^ 1] = 0u;
    cnt[CNT_FETCH] = 0u;
    cnt[CNT_LOOP_FETCH] = 0u;
    seen[0] = taken ? q : 0u;
    seen[1] = q;
    __threadfence_system();
}

gr_status bounce_begin(const BounceReadback& rb, uint32_t* cnt, uint32_t depth, uint32_t take, cudaStream_t st) {
    const uint32_t k = depth & 3;
    k_bounce_begin<<<1, 1, 0, st>>>(cnt, static_cast<int>(depth & 1), take, rb.host + 2 * k);
    GR_CUDA_TRY(cudaGetLastError());
    GR_CUDA_TRY(cudaEventRecord(rb.ev[k], st));
    return GR_OK;
}

// What the host knows of a group's queue: `bound`, an upper bound of its current length (a
// queue only gets shorter), and the length expected at the next bounce, which falls about
// as it fell last.
struct QueueOutlook {
    uint32_t bound;
    uint64_t expected;
    explicit QueueOutlook(uint32_t n) : bound(n), expected(n) {}
    // Whether to offer the next bounce's queue to the path loop: a launch that finds it too
    // long costs about 5 us, one left out on a short queue 30 us and more.
    bool offer() const { return expected <= PATH_LOOP_MAX + PATH_LOOP_MAX / 2 || bound <= PATH_LOOP_MAX; }
};

// Waits for what bounce `depth` began with (the bounce itself still runs); `more`: false when
// it was the last one.
gr_status bounce_wait(const BounceReadback& rb, uint32_t depth, QueueOutlook& out, bool& more) {
    const uint32_t k = depth & 3;
    GR_CUDA_TRY(cudaEventSynchronize(rb.ev[k]));
    const uint32_t before = out.bound, seen = rb.host[2 * k + 1];
    out.bound = seen;
    out.expected = before ? static_cast<uint64_t>(seen) * seen / before : 0u;
    more = rb.host[2 * k] == 0 && seen != 0;
    return GR_OK;
}

// `fetch`: the kernel's ray counter, zero before the launch.
template <int W, bool COUNT>
gr_status extend_launch(const DeviceScene& s, uint32_t cap_n, const uint32_t* count, const float4* qo,
                        const float4* qd, float4* qh, int* err, unsigned long long* rays, uint32_t* fetch,
                        cudaStream_t st, bool one_origin) {
    const size_t smem = step_stack_smem_bytes(BLOCK);
    const int grid = resident_grid(k_extend_refill<W, COUNT>, smem, cap_n);
    k_extend_refill<W, COUNT><<<grid, BLOCK, smem, st>>>(s, count, qo, qd, qh, err, rays, fetch, one_origin);
    return GR_OK;
}

// one_origin: every ray of the queue starts at qo[0] (see k_extend_refill).
gr_status extend_any(const DeviceScene& s, bool count_traversal, uint32_t cap_n, const uint32_t* count,
                     const float4* qo, const float4* qd, float4* qh, int* err, unsigned long long* rays,
                     uint32_t* fetch, cudaStream_t st, bool one_origin) {
    const bool o1 = one_origin;
    if (count_traversal) {
        switch (s.width) {
            case 2: return extend_launch<2, true>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
            case 4: return extend_launch<4, true>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
            default: return extend_launch<8, true>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
        }
    }
    switch (s.width) {
        case 2: return extend_launch<2, false>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
        case 4: return extend_launch<4, false>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
        default: return extend_launch<8, false>(s, cap_n, count, qo, qd, qh, err, rays, fetch, st, o1);
    }
}

}  // namespace
}  // namespace gr
