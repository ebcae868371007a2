// Closest-hit and shadow traversal of the wide BVH (replaces Bvh::intersect,
// geom/bvh.rs:406-456, and Bvh::visibility, bvh.rs:460-477).
//
// One thread per ray.  A node is 2W float4s (W = 2, 4, 8) read with vector loads;
// every child box is slab-tested (far distances inflated by 1 + 2 gamma(3) as in
// core/bbox.rs:78-113), the hit children are ordered near-to-far by a sorting network
// on (distance | slot) keys, and the farther ones go on a per-thread stack of
// (child, entry distance) pairs: the first SMEM_STACK entries in shared memory, column
// `threadIdx.x`, deeper ones in a local array.  Popped entries whose entry distance is
// no longer below the closest hit are skipped.  Every traversal (closest hit, shadow
// rays, query kernels) runs the step functions below: visit_node and visit_leaf, one ray per
// lane, or trace_grouped, which makes the same tests with W lanes per ray.
// Leaves hold up to 16 consecutive primitive records.  The primitive tests are the
// reference's Moller-Trumbore (geom/mesh.rs:270-308) and sphere quadratic
// (geom/sphere.rs:70-101) with the same operation order, so a hit distance is
// bit-identical to the reference's for the same triangle.
#pragma once

#include "scene.hpp"

namespace gr {

struct TraceResult {
    float t;
    int32_t k;  // leaf-order primitive index, -1 = miss
    float u, v;
};

// Reference primitive tests.  Returns the distance (0 = miss).
GR_D float intersect_prim(const float4 p0, const float4 p1, const float4 p2, V3 o, V3 d, float& uo, float& vo) {
    if (__float_as_int(p2.w) == PRIM_TRIANGLE) {
        V3 c = V3{p0.x, p0.y, p0.z};
        V3 e1 = V3{p1.x, p1.y, p1.z};
        V3 e2 = V3{p2.x, p2.y, p2.z};
        V3 p = cross(d, e2);
        float det = dot(e1, p);
        if (nearly_zero(det)) return 0.0f;
        float inv_det = 1.0f / det;
        V3 t = o - c;
        float u = dot(t, p) * inv_det;
        if (u < 0.0f || u > 1.0f) return 0.0f;
        V3 q = cross(t, e1);
        float v = dot(d, q) * inv_det;
        if (v < 0.0f || (u + v) > 1.0f) return 0.0f;
        float dist = dot(e2, q) * inv_det;
        if (!is_positive(dist)) return 0.0f;
        uo = u;
        vo = v;
        return dist;
    }
    V3 oc = o - V3{p0.x, p0.y, p0.z};
    float r = p1.x;
    float a = dot(d, d);
    float b = dot(d, oc);
    float c = dot(oc, oc) - (r * r);
    float disc = (b * b) - (a * c);
    if (disc > 0.0f) {
        float sq = sqrtf(disc);
        float res_pos = -b + sq;
        float res_neg = -b - sq;
        if (is_positive(res_neg)) return res_neg;
        if (is_positive(res_pos)) return res_pos;
    }
    return 0.0f;
}

// child[slot] without dynamic register indexing (keeps the node in registers).
template <int W>
GR_D int32_t select_child(const float (&f)[8 * W], uint32_t slot) {
    int32_t r = 0;
#pragma unroll
    for (int j = 0; j < W; ++j)
        if (static_cast<uint32_t>(j) == slot) r = __float_as_int(f[6 * W + j]);
    return r;
}

template <int N>
GR_D void sort_keys(uint32_t (&k)[N]) {
    // Odd-even transposition network, fully unrolled (N <= 8).
#pragma unroll
    for (int pass = 0; pass < N; ++pass) {
#pragma unroll
        for (int i = pass & 1; i + 1 < N; i += 2) {
            uint32_t a = k[i], b = k[i + 1];
            k[i] = min(a, b);
            k[i + 1] = max(a, b);
        }
    }
}

}  // namespace gr

namespace gr {

// ---------------------------------------------------------------------------
// Step-wise traversal for the persistent extension kernel.  The state of one ray lives
// in registers; trav_step() processes one interior node or one leaf.  The stack keeps
// its first SMEM_STACK entries in this thread's shared-memory column and spills deeper
// entries to a per-thread local array (rarely touched, cached in L1), so the shared
// footprint no longer scales with the tree's worst-case depth.
// Stack entries per thread kept in shared memory (MAX_STACK in common.cuh: both builds
// reject deeper trees); deeper entries go to the local spill array.  On the path-tracer
// workload (102,422 triangles, 1024 x 1024, 64 spp) 4 / 8 / 12 / 16 measured 1863 /
// 1883 / 1887 / 1881 Msamples/s: the L1 left to node and primitive loads by a smaller
// shared part does not matter.
#ifndef GR_SMEM_STACK
#define GR_SMEM_STACK 16
#endif
constexpr int SMEM_STACK = GR_SMEM_STACK;
static_assert(SMEM_STACK >= 1 && SMEM_STACK <= MAX_STACK, "shared stack part within the stack bound");

// A warp tracing rays from a queue (trace_queue) takes new rays for its idle lanes once
// EXTEND_REFILL of them are idle, and tests leaves once EXTEND_LEAVES of its lanes stand at
// one (or none stands at a node), not whenever one does: a step runs either the node test
// or the leaf test for the whole warp.  On the path-tracer workload (102,422 triangles,
// 1024 x 1024, 64 spp) testing leaves at once took 15.3 ms of extension per render, and
// waiting for 4 / 6 / 8 / 12 lanes 15.2 / 14.4 / 14.3 / 15.1 (refilling at 16); refilling
// at 8 / 12 / 16 / 20 / 24 (waiting for 8) 15.7 / 14.7 / 14.3 / 14.1 / 14.4.
constexpr int EXTEND_REFILL = 20;
constexpr int EXTEND_LEAVES = 8;

// What a traversal step reads.  A kernel whose lanes trace rays of different scenes keeps
// one per lane in registers instead of reloading it through a scene record at every step.
struct TraceScene {
    const float4* nodes;
    const float4* prims;
    uint32_t step_budget;
};

struct TravState {
    V3 o, d, inv;
    float closest;
    float hu, hv;
    int32_t ref;
    int32_t hit;
    int sp;
    bool nx, ny, nz;
};

GR_D void trav_init(TravState& t, V3 o, V3 d, float t_max) {
    t.o = o;
    t.d = d;
    t.inv = V3{1.0f / d.x, 1.0f / d.y, 1.0f / d.z};
    t.nx = d.x < 0.0f;
    t.ny = d.y < 0.0f;
    t.nz = d.z < 0.0f;
    t.closest = t_max;
    t.hu = t.hv = 0.0f;
    t.ref = 0;
    t.hit = -1;
    t.sp = 0;
}

// Stack entries are (child reference, entry distance bits) pairs, one 64-bit access each.
// STRIDE: threads of the block, so that an entry's address is the column's plus a
// constant shift.
template <int STRIDE>
struct StackView {
    int2* s;      // this thread's shared column
    int2* spill;  // local overflow, MAX_STACK - SMEM_STACK entries
    static constexpr int stride = STRIDE;
    GR_D int2* at(int sp) const { return s + sp * STRIDE; }
    GR_D void push(int sp, int32_t ref, uint32_t te_bits) const {
        const int2 e = make_int2(ref, static_cast<int>(te_bits));
        if (sp < SMEM_STACK) s[sp * STRIDE] = e;
        else spill[sp - SMEM_STACK] = e;
    }
    GR_D void pop(int sp, int32_t& ref, float& te) const {
        int2 e;
        if (sp < SMEM_STACK) e = s[sp * STRIDE];  // shared and local loads kept apart
        else e = spill[sp - SMEM_STACK];
        ref = e.x;
        te = __int_as_float(e.y);
    }
};

constexpr uint32_t KEY_MISS = 0xFFFFFFFFu;  // sorts after every hit child

// One comparator of the sorting network at width 4, each key with its child reference.
GR_D void order_pair(uint32_t& ka, uint32_t& kb, int32_t& ra, int32_t& rb) {
    const bool swap = kb < ka;
    const uint32_t k = swap ? kb : ka;
    kb = swap ? ka : kb;
    ka = k;
    const int32_t r = swap ? rb : ra;
    rb = swap ? ra : rb;
    ra = r;
}

// Tests one wide node against the ray: pushes the far hit children (sorted by entry
// distance, nearest last) and makes the nearest hit child the current reference.
// Returns false when no child is hit.  A push beyond MAX_STACK sets *err = 1 and
// `overflow`.
template <int W, bool COUNT, class S, class K>
GR_D bool visit_node(const S& s, TravState& t, const K& stk, int* err, uint32_t* counts,
                     bool& overflow) {
    const float inflate = 1.0f + 2.0f * gamma_n(3.0f);
    if (COUNT) counts[0] += 1;
    const float4* nb = s.nodes + static_cast<size_t>(t.ref) * (2 * W);
    // f holds the rows lo_x lo_y lo_z hi_x hi_y hi_z child (W floats each).  With W a
    // multiple of 4 a row is whole float4s, so the ray loads its near and far planes
    // straight into the lo and hi rows (row offsets from its direction signs) and skips
    // the padding row: no per-child selects, one load fewer.  The arithmetic is the same
    // as selecting them.
    float f[8 * W];
    if (W % 4 == 0) {
        constexpr int R = W / 4;  // float4 per row
        const int rows[7] = {t.nx ? 3 : 0, t.ny ? 4 : 1, t.nz ? 5 : 2, t.nx ? 0 : 3, t.ny ? 1 : 4, t.nz ? 2 : 5, 6};
#pragma unroll
        for (int r = 0; r < 7; ++r)
#pragma unroll
            for (int q = 0; q < R; ++q) {
                float4 x = __ldg(nb + rows[r] * R + q);
                f[r * W + 4 * q] = x.x;
                f[r * W + 4 * q + 1] = x.y;
                f[r * W + 4 * q + 2] = x.z;
                f[r * W + 4 * q + 3] = x.w;
            }
    } else {
#pragma unroll
        for (int q = 0; q < 2 * W; ++q) {
            float4 x = __ldg(nb + q);
            f[4 * q] = x.x;
            f[4 * q + 1] = x.y;
            f[4 * q + 2] = x.z;
            f[4 * q + 3] = x.w;
        }
    }
    uint32_t key[W];
    int h = 0;
    // The slab test (tmin <= tmax, tmax > 0, tmin < closest) on te = max(tmin, 0): the same
    // result (closest > 0), except that a box whose far distance is exactly 0 counts as
    // hit, which can only add a node to visit.
    auto child_key = [&](int j, float tmin, float tmax) {
        const float te = fmaxf(tmin, 0.0f);
        const bool hit = te <= tmax && te < t.closest;
        key[j] = hit ? ((__float_as_uint(te) & ~7u) | static_cast<uint32_t>(j)) : KEY_MISS;
        h += hit ? 1 : 0;
    };
    if (W % 4 == 0) {  // rows 0-2 near, 3-5 far; two children per packed operation
        const F2 nox = pack2(-t.o.x, -t.o.x), noy = pack2(-t.o.y, -t.o.y), noz = pack2(-t.o.z, -t.o.z);
        const F2 ix = pack2(t.inv.x, t.inv.x), iy = pack2(t.inv.y, t.inv.y), iz = pack2(t.inv.z, t.inv.z);
        auto plane = [&](int row, int j, F2 no, F2 inv, float& a, float& b) {
            unpack2(mul2(add2(pack2(f[row * W + j], f[row * W + j + 1]), no), inv), a, b);
        };
#pragma unroll
        for (int j = 0; j < W; j += 2) {
            float ax, bx, ay, by, az, bz;
            plane(0, j, nox, ix, ax, bx);
            plane(1, j, noy, iy, ay, by);
            plane(2, j, noz, iz, az, bz);
            const float na = fmaxf(fmaxf(ax, ay), az), nb2 = fmaxf(fmaxf(bx, by), bz);
            plane(3, j, nox, ix, ax, bx);
            plane(4, j, noy, iy, ay, by);
            plane(5, j, noz, iz, az, bz);
            float fa, fb;
            unpack2(mul2(pack2(fminf(fminf(ax, ay), az), fminf(fminf(bx, by), bz)), pack2(inflate, inflate)), fa, fb);
            child_key(j, na, fa);
            child_key(j + 1, nb2, fb);
        }
    } else {
#pragma unroll
        for (int j = 0; j < W; ++j) {
            float lx = f[0 * W + j], ly = f[1 * W + j], lz = f[2 * W + j];
            float hx = f[3 * W + j], hy = f[4 * W + j], hz = f[5 * W + j];
            float t0x = ((t.nx ? hx : lx) - t.o.x) * t.inv.x;
            float t1x = ((t.nx ? lx : hx) - t.o.x) * t.inv.x;
            float t0y = ((t.ny ? hy : ly) - t.o.y) * t.inv.y;
            float t1y = ((t.ny ? ly : hy) - t.o.y) * t.inv.y;
            float t0z = ((t.nz ? hz : lz) - t.o.z) * t.inv.z;
            float t1z = ((t.nz ? lz : hz) - t.o.z) * t.inv.z;
            child_key(j, fmaxf(fmaxf(t0x, t0y), t0z), fminf(fminf(t1x, t1y), t1z) * inflate);
        }
    }
    // Width 4: the 5-comparator network with the child references carried along (instead
    // of picked by the sorted slots: the path loop's meshes 0.996 -> 0.944 ms), and one
    // bounds test for all pushes.
    if (W == 4) {
        int32_t c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = __float_as_int(f[6 * W + j % W]);
        order_pair(key[0], key[1], c[0], c[1]);
        order_pair(key[2], key[3 % W], c[2], c[3]);
        order_pair(key[0], key[2], c[0], c[2]);
        order_pair(key[1], key[3 % W], c[1], c[3]);
        order_pair(key[1], key[2], c[1], c[2]);
        if (key[0] == KEY_MISS) return false;
        const int n = (key[1] != KEY_MISS ? 1 : 0) + (key[2] != KEY_MISS ? 1 : 0) + (key[3 % W] != KEY_MISS ? 1 : 0);
        const int top = t.sp + n;
        if (top <= SMEM_STACK) {
            int2* e = stk.at(top);
            if (key[1] != KEY_MISS) e[-K::stride] = make_int2(c[1], static_cast<int>(key[1] & ~7u));
            if (key[2] != KEY_MISS) e[-2 * K::stride] = make_int2(c[2], static_cast<int>(key[2] & ~7u));
            if (key[3 % W] != KEY_MISS) e[-3 * K::stride] = make_int2(c[3], static_cast<int>(key[3 % W] & ~7u));
        } else if (top <= MAX_STACK) {
#pragma unroll
            for (int j = 3; j >= 1; --j)
                if (key[j % W] != KEY_MISS) stk.push(top - j, c[j], key[j % W] & ~7u);
        } else {
            *err = 1;
            overflow = true;
            return false;
        }
        t.sp = top;
        t.ref = c[0];
        return true;
    }
    if (h == 0) return false;
    sort_keys<W>(key);
    if (t.sp + h - 1 > MAX_STACK) {
        *err = 1;
        overflow = true;
        return false;
    }
#pragma unroll
    for (int j = W - 1; j >= 1; --j) {
        if (j < h) {
            stk.push(t.sp, select_child<W>(f, key[j] & 7u), key[j] & ~7u);
            ++t.sp;
        }
    }
    t.ref = select_child<W>(f, key[0] & 7u);
    return true;
}

// Intersects the primitives of leaf `ref`, keeping the closest hit in t.  With ANY_HIT
// it returns true at the first hit closer than t.closest.
template <bool ANY_HIT, bool COUNT, class S>
GR_D bool visit_leaf(const S& s, TravState& t, int32_t ref, uint32_t* counts) {
    uint32_t enc = ~static_cast<uint32_t>(ref);
    uint32_t first = enc >> LEAF_COUNT_BITS;
    uint32_t count = (enc & (MAX_LEAF_PRIMS - 1)) + 1;
    if (COUNT) counts[1] += count;
    for (uint32_t k = first; k < first + count; ++k) {
        const float4* pr = s.prims + 3 * static_cast<size_t>(k);
        float4 p0 = __ldg(pr), p1 = __ldg(pr + 1), p2 = __ldg(pr + 2);
        float u, v;
        float dist = intersect_prim(p0, p1, p2, t.o, t.d, u, v);
        if (dist != 0.0f && dist < t.closest) {
            t.closest = dist;
            t.hit = static_cast<int32_t>(k);
            t.hu = u;
            t.hv = v;
            if (ANY_HIT) return true;
        }
    }
    return false;
}

// Pops the next stacked child that can still hold a closer hit into t.ref.  Returns
// false when the stack is exhausted.
template <class K>
GR_D bool pop_next(TravState& t, const K& stk) {
    while (t.sp > 0) {
        --t.sp;
        int32_t r;
        float te;
        stk.pop(t.sp, r, te);
        if (te < t.closest) {
            t.ref = r;
            return true;
        }
    }
    return false;
}

// One traversal step towards the closest hit.  Returns true when the ray is finished (t.hit
// / t.closest hold the hit).
// S is DeviceScene or TraceScene: the step functions read only `nodes` and `prims`.
template <int W, class S, class K>
GR_D bool trav_step(const S& s, TravState& t, const K& stk, int* err) {
    if (t.ref >= 0) {
        bool overflow = false;
        const bool descended = visit_node<W, false>(s, t, stk, err, nullptr, overflow);
        if (overflow) {
            t.hit = -1;
            return true;
        }
        if (descended) return false;
    } else {
        visit_leaf<false, false>(s, t, t.ref, nullptr);
    }
    return !pop_next(t, stk);
}

GR_HD constexpr size_t step_stack_smem_bytes(int threads) {
    return static_cast<size_t>(SMEM_STACK) * threads * (sizeof(int32_t) + sizeof(float));
}

// A thread's traversal stack: its column of the block's shared stack (dynamic shared
// memory starting at `smem`, step_stack_smem_bytes(STRIDE) bytes, STRIDE = blockDim.x) and its local
// spill array.
template <int STRIDE>
GR_D StackView<STRIDE> thread_stack(unsigned char* smem, int2* spill) {
    return StackView<STRIDE>{reinterpret_cast<int2*>(smem) + threadIdx.x, spill};
}

// ---------------------------------------------------------------------------
// A lane's scene, held by lane `src`.
GR_D TraceScene scene_of(const TraceScene& s, int src) {
    return TraceScene{reinterpret_cast<const float4*>(
                          __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(s.nodes), src)),
                      reinterpret_cast<const float4*>(
                          __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(s.prims), src)),
                      __shfl_sync(0xffffffffu, s.step_budget, src)};
}
GR_D TraceScene scene_of(const DeviceScene& s, int) { return TraceScene{s.nodes, s.prims, s.step_budget}; }

// Scenes of at least this many components have a warp's last rays traced by groups of
// lanes (trace_grouped): 1,437 -> 1,386 us on 641 x 359 x 9 spp of 12,000 triangles, 293 ->
// 278 on 64 x 64 x 2 spp of 50,000.  The few steps of a ray in a small scene do not repay
// the hand-over (Cornell box 128 x 128 x 4 spp: 220 -> 230, BDPT 795 -> 813).
constexpr uint32_t GROUPED_COMPONENTS = 1024;

// Closest hits (ANY_HIT: any) of the rays of the lanes in `mask` (at most 32 / W), W lanes each: a lane
// tests one child of a node or one primitive of a leaf.  The same tests, order and hits as
// trav_step, whose some 250 dependent instructions per node are what a ray alone in its warp
// waits for.  `steps` counts on; a ray whose stack would outgrow its shared part is given
// back unfinished (deep), one that runs out of steps with `over` set; the others end.  Every
// lane of the warp calls it with the same mask.
template <int W, bool ANY_HIT, class S, class K>
GR_D void trace_grouped(unsigned mask, const S& scene, TravState& t, uint32_t& steps, const K& stk, bool& deep,
                        bool& over) {
    constexpr unsigned all = 0xffffffffu, ones = (1u << W) - 1u;
    const unsigned lane = threadIdx.x & 31u, j = lane % W, g0 = lane - j;
    const float inflate = 1.0f + 2.0f * gamma_n(3.0f);
    unsigned rest = mask;
    for (unsigned k = 0; k < lane / W; ++k) rest &= rest - 1u;
    bool on = rest != 0u, out = false, late = false;
    const int src = on ? __ffs(rest) - 1 : static_cast<int>(lane);
    const TraceScene s = scene_of(scene, src);
    auto of = [&](float x) { return __shfl_sync(all, x, src); };
    const V3 o = V3{of(t.o.x), of(t.o.y), of(t.o.z)}, d = V3{of(t.d.x), of(t.d.y), of(t.d.z)};
    const V3 inv = V3{of(t.inv.x), of(t.inv.y), of(t.inv.z)};
    float closest = of(t.closest), hu = of(t.hu), hv = of(t.hv);
    int32_t ref = __shfl_sync(all, t.ref, src), hit = __shfl_sync(all, t.hit, src);
    int sp = __shfl_sync(all, t.sp, src);
    uint32_t n = __shfl_sync(all, steps, src);
    // Rows of this lane's child: near and far planes by the ray's direction signs.
    const uint32_t xn = (d.x < 0.0f ? 3 : 0) * W + j, xf = (d.x < 0.0f ? 0 : 3) * W + j;
    const uint32_t yn = (d.y < 0.0f ? 4 : 1) * W + j, yf = (d.y < 0.0f ? 1 : 4) * W + j;
    const uint32_t zn = (d.z < 0.0f ? 5 : 2) * W + j, zf = (d.z < 0.0f ? 2 : 5) * W + j;
    int2* col = stk.at(0) + (src - static_cast<int>(lane));
    // The next stacked child that can hold a closer hit, as pop_next.
    auto next = [&](bool want) {
        bool found = false;
        while (want && !found && sp > 0) {
            --sp;
            const int2 e = col[sp * K::stride];
            found = __int_as_float(e.y) < closest;
            ref = e.x;
        }
        if (want && !found) on = false;
    };
    __syncwarp();
    for (;;) {
        if (on && n > s.step_budget) {
            on = false;
            late = true;
        }
        if (on && sp + W - 1 > SMEM_STACK) {
            on = false;
            out = true;
        }
        if (!__any_sync(all, on)) break;
        const bool node = on && ref >= 0;
        if (__any_sync(all, node)) {
            uint32_t key = KEY_MISS;
            int32_t child = 0;
            if (node) {
                const float* f = reinterpret_cast<const float*>(s.nodes + static_cast<size_t>(ref) * (2 * W));
                const float ax = __ldg(f + xn), ay = __ldg(f + yn), az = __ldg(f + zn);
                const float bx = __ldg(f + xf), by = __ldg(f + yf), bz = __ldg(f + zf);
                child = __float_as_int(__ldg(f + 6 * W + j));
                const float tmin = fmaxf(fmaxf((ax - o.x) * inv.x, (ay - o.y) * inv.y), (az - o.z) * inv.z);
                const float tmax = fminf(fminf((bx - o.x) * inv.x, (by - o.y) * inv.y), (bz - o.z) * inv.z) * inflate;
                const float te = fmaxf(tmin, 0.0f);
                if (te <= tmax && te < closest) key = (__float_as_uint(te) & ~7u) | j;
                ++n;
            }
            uint32_t rank = 0;
#pragma unroll
            for (int x = 1; x < W; ++x) rank += __shfl_xor_sync(all, key, x) < key ? 1u : 0u;
            const unsigned hits = (__ballot_sync(all, key != KEY_MISS) >> g0) & ones;
            const unsigned first = (__ballot_sync(all, key != KEY_MISS && rank == 0u) >> g0) & ones;
            const int32_t near = __shfl_sync(all, child, static_cast<int>(g0) + (first ? __ffs(first) - 1 : 0));
            const int far = __popc(hits) - 1;
            __syncwarp();  // every lane of the group has read the entries that are written over (next)
            if (key != KEY_MISS && rank > 0u)
                col[(sp + far - static_cast<int>(rank)) * K::stride] = make_int2(child, static_cast<int>(key & ~7u));
            if (node && hits) {
                sp += far;
                ref = near;
            }
            __syncwarp();
            next(node && !hits);
        }
        const bool leaf = on && ref < 0;
        if (__any_sync(all, leaf)) {
            const uint32_t enc = ~static_cast<uint32_t>(ref), at = enc >> LEAF_COUNT_BITS;
            const uint32_t count = leaf ? (enc & (MAX_LEAF_PRIMS - 1)) + 1 : 0u;
            for (uint32_t b = 0; __any_sync(all, b < count); b += W) {
                float dist = 0.0f, u = 0.0f, v = 0.0f;
                if (b + j < count) {
                    const float4* pr = s.prims + 3 * static_cast<size_t>(at + b + j);
                    dist = intersect_prim(__ldg(pr), __ldg(pr + 1), __ldg(pr + 2), o, d, u, v);
                }
                float best = dist != 0.0f && dist < closest ? dist : FLT_MAX;
                const float mine = best;
#pragma unroll
                for (int x = 1; x < W; x <<= 1) best = fminf(best, __shfl_xor_sync(all, best, x));
                const unsigned won = (__ballot_sync(all, mine == best && best < FLT_MAX) >> g0) & ones;
                const int w = static_cast<int>(g0) + (won ? __ffs(won) - 1 : 0);
                u = __shfl_sync(all, u, w);
                v = __shfl_sync(all, v, w);
                if (won) {
                    closest = best;
                    hit = static_cast<int32_t>(at + b) + (w - static_cast<int>(g0));
                    hu = u;
                    hv = v;
                }
            }
            if (leaf) {
                ++n;
                if (ANY_HIT && hit >= 0) on = false;
            }
            next(leaf && on);
        }
    }
    __syncwarp();
    const int from = static_cast<int>(W * __popc(mask & ((1u << lane) - 1u))) & 31;
    const float fc = __shfl_sync(all, closest, from), fu = __shfl_sync(all, hu, from), fv = __shfl_sync(all, hv, from);
    const int32_t fr = __shfl_sync(all, ref, from), fh = __shfl_sync(all, hit, from);
    const int fs = __shfl_sync(all, sp, from);
    const uint32_t fn = __shfl_sync(all, n, from);
    const int state = __shfl_sync(all, (out ? 1 : 0) | (late ? 2 : 0), from);
    if ((mask >> lane) & 1u) {
        t.closest = fc;
        t.hu = fu;
        t.hv = fv;
        t.ref = fr;
        t.hit = fh;
        t.sp = fs;
        steps = fn;
        deep = state & 1;
        over = state & 2;
    }
}

// ---------------------------------------------------------------------------
// Queue traversal: a warp keeps its lanes busy across rays q = 0 .. n - 1.
//   grab(k, lane)    the first of the next k rays (a counter shared by the whole grid or
//                    by the warp alone; rays >= n are not there)
//   load(q, t)       starts ray q (trav_init), or returns false when nothing is to trace
//   scene()          this lane's scene: nodes, prims and step budget
//   store(q, t)      the finished ray: t.hit / t.closest / t.hu / t.hv
// Each iteration every busy lane that is at a node, or else every one that is at a leaf,
// takes one traversal step (see EXTEND_LEAVES); once enough lanes are idle, the warp
// grabs that many rays and hands them to its idle lanes.  So a lane whose ray ended early
// starts another one, instead of idling until the warp's longest ray ends.  A ray that
// takes more than its scene's step budget is abandoned as a miss: *err = 2 and, if err_ray
// is given, its index there.  With ANY_HIT a ray ends at its first hit.  `grouped` (with
// GROUPED, and no COUNT): once no rays are left to grab, a warp's last ones are traced by groups of
// lanes.
//
// Every warp intrinsic runs where control flow is warp-uniform: the loop's iterations are
// the same for all lanes, the refill condition depends on ballot results and on the
// grabbed base only, and the loop ends on a ballot.  It terminates: an iteration steps at
// least one busy lane (each ray has the step budget, and each ray is handed out once), or
// finds every lane idle, refills and gets rays or learns that none are left.
//
// Bound by instruction issue (71-77% active) and the L1 data pipe (54-67%: 112 bytes per
// lane and node) on camera rays and first bounces, by node-load latency further on.
template <int W, bool ANY_HIT, bool COUNT, bool GROUPED = false, class K, class Grab, class SceneOf, class Load,
          class Store>
GR_D void trace_queue(uint32_t n, const K& stk, int* err, int* err_ray, uint32_t* counts, const Grab& grab,
                      const SceneOf& scene, const Load& load, const Store& store, bool grouped = false) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    TravState t;
    uint32_t q = 0, steps = 0;
    bool busy = false, exhausted = false, deep = false;  // deep: grouped lanes gave this ray back
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !busy);
        if (!exhausted && __popc(idle) >= EXTEND_REFILL) {
            const uint32_t base = grab(static_cast<uint32_t>(__popc(idle)), lane);
            exhausted = static_cast<uint64_t>(base) + __popc(idle) >= n;
            if (!busy) {
                q = base + __popc(idle & below);
                if (q < n) {
                    busy = load(q, t);
                    steps = 0;
                    deep = false;
                }
            }
        }
        if (GROUPED && grouped && exhausted) {
            const unsigned last = __ballot_sync(0xffffffffu, busy && !deep);
            if (last && __popc(last) <= 32 / W) {
                bool over = false;
                trace_grouped<W, ANY_HIT>(last, scene(), t, steps, stk, deep, over);
                if (over) {
                    atomicExch(err, 2);
                    if (err_ray) atomicExch(err_ray, static_cast<int>(q));
                    t.hit = -1;
                }
                if (((last >> lane) & 1u) && !deep) {
                    store(q, t);
                    busy = false;
                }
                continue;
            }
        }
        const bool leaf = busy && t.ref < 0, node = busy && t.ref >= 0;
        const unsigned leaves = __ballot_sync(0xffffffffu, leaf), nodes = __ballot_sync(0xffffffffu, node);
        if ((leaves | nodes) == 0u) {  // every lane idle: grab again, or none is left
            if (exhausted) break;
            continue;
        }
        bool pop = false, done = false;
        // The last rays of a warp wait for no more than a quarter of it: 512 x 512 x 4 spp of
        // 102,400 triangles 1,171 -> 1,144 us, 1024 x 1024 x 64 spp 24.24 -> 24.16 ms.
        const int enough = exhausted ? min(EXTEND_LEAVES, max(1, __popc(leaves | nodes) / 4)) : EXTEND_LEAVES;
        if (nodes == 0u || __popc(leaves) >= enough) {
            if (leaf) {
                done = visit_leaf<ANY_HIT, COUNT>(scene(), t, t.ref, counts);
                pop = !done;
                ++steps;
            }
        } else if (node) {
            bool overflow = false;
            pop = !visit_node<W, COUNT>(scene(), t, stk, err, counts, overflow);
            ++steps;
            if (overflow) {
                t.hit = -1;
                done = true;
                pop = false;
            }
        }
        if (pop) done = !pop_next(t, stk);
        if (busy) {
            if (!done && steps > scene().step_budget) {
                atomicExch(err, 2);
                if (err_ray) atomicExch(err_ray, static_cast<int>(q));
                t.hit = -1;
                done = true;
            }
            if (done) {
                store(q, t);
                busy = false;
            }
        }
    }
}

// Rays handed out from a counter in global memory, zero before the launch: one atomic per
// refill.
struct SharedCounter {
    uint32_t* next;
    GR_D uint32_t operator()(uint32_t k, unsigned lane) const {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(next, k);
        return __shfl_sync(0xffffffffu, base, 0);
    }
};

}  // namespace gr
