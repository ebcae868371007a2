// Pieces shared by the wavefront integrators (pt.cu, bdpt.cu): the extension kernel
// over a compacted ray queue, the warp-aggregated queue push and grid sizing.
#pragma once

#include <algorithm>
#include <cstdlib>

#include "path_loop.cuh"
#include "runtime.hpp"
#include "shade_sort.cuh"
#include "traverse.cuh"


namespace gr {
namespace {

constexpr int BLOCK = 128;

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

// Grid of a path-loop kernel for at most `most` paths; `smem` is the block's.
template <class K>
gr_status path_loop_grid(K kernel, size_t smem, uint32_t most, int& grid) {
    if (smem > 48 * 1024) GR_CUDA_TRY(allow_sort_smem(kernel, smem));
    grid = resident_grid(kernel, smem, (most + PATH_LOOP_MIN_LANES - 1) / PATH_LOOP_MIN_LANES * 32u, PATH_LOOP_THREADS);
    return GR_OK;
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
