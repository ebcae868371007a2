// Wavefront BDPT: BdptIntegrator::integrate (render/integrators.rs:357-418) with the
// reference's uniform strategy weights 1 / (c + l) (integrators.rs:345-354), and two
// extensions (off by default): power-heuristic MIS weights and the light-tracing
// strategy (light-walk vertex -> pinhole camera, splatted with atomics).
//
//   raygen    per path: jitter + camera ray (camera walk, slot 2i) and Bvh::sample_light
//             + the light vertex (light walk, slot 2i+1), both pushed to one queue
//   extend    closest hit (shared with the path tracer)
//   (once few walks are left, or from the start, one launch carries them to their end)
//   shade     random_walk (integrators.rs:138-229) for both walks: Material::sample_world,
//             throughput, shading-normal correction on light paths, roulette from
//             length rr_len; each surface vertex is stored (an escape connects to nothing)
//   order     paths counting-sorted by (camera, light) walk length; the strategies of all
//             paths laid out as items, all paths of one strategy (c, l) next to each other
//   connect   per item, connect() (integrators.rs:269-343) without the visibility test,
//             times its weight; terms that need one queue a shadow ray
//   light_trace  with light tracing, every light-walk vertex inside the image gets a
//             camera term (its own items and kernel)
//   shadow    Bvh::visibility (bvh.rs:460-477) as an any-hit query
//   gather    per path, sums the weighted strategy terms in the reference's loop order
//             (deterministic)
//   splat     visible light-tracing terms are added to the film's splat buffer, with atomics
//   film      the deterministic splat of film.cu
#include <algorithm>
#include <cstdlib>

#include "path_order.cuh"
#include "runtime.hpp"
#include "shade_sort.cuh"
#include "wavefront.cuh"

namespace gr {

namespace {

constexpr int VREC = 8;            // float4 per stored vertex
constexpr uint32_t F_SKIP = 1;     // light sample had a zero pdf: the reference returns early
constexpr uint32_t F_ESCAPE = 2;   // the camera walk escaped (environment term)
constexpr float E_NO_TEST = 0.0f;  // entry flags (float in .w)
constexpr float E_PENDING = 1.0f;
constexpr float E_VISIBLE = 2.0f;
constexpr float E_OCCLUDED = 3.0f;
constexpr int CNT_SHADOWQ = 13;
constexpr int CNT_SHADOWF = 14;  // shadow rays handed out

// The pinhole camera seen from the scene (light-tracing and MIS extensions): position,
// world directions of its x, y, z axes (the camera matrix is a rotation and a
// translation, camera.rs:42-61) and the [-1, 1]^2 window on the plane at distance 1.
struct PinholeView {
    V3 pos, axis[3];
    float wx, wy, area;
    // Film position (s, t) of p, its distance and the cosine between the viewing axis
    // and the direction to p; false when p is behind the camera or outside the window.
    GR_D bool project(V3 p, float& s, float& t, float& dist, float& cos_view) const {
        V3 v = p - pos;
        float cx = dot(v, axis[0]), cy = dot(v, axis[1]), cz = dot(v, axis[2]);
        if (!(cz < 0.0f)) return false;
        s = (cx / -cz) / wx;
        t = (cy / -cz) / wy;
        dist = magnitude(v);
        cos_view = -cz / dist;
        return s >= -1.0f && s <= 1.0f && t >= -1.0f && t <= 1.0f;
    }
    // Solid-angle pdf of a camera ray spread uniformly over the window: 1 / (area cos^3).
    GR_D float dir_pdf(float cos_view) const { return 1.0f / (area * cos_view * cos_view * cos_view); }
};

struct BdptParams {
    DevCamera cam;
    PinholeView view;
    PathOrder order;  // which sample a path is
    uint32_t width, height, first_pass;
    uint64_t seed;
    uint32_t max_len, rr_len;
    uint32_t n;       // paths in this group
    uint32_t nslots;  // 2 n
    uint32_t mis;     // power-heuristic weights (else uniform)
    uint32_t lt;      // light-tracing strategy
};

// Solid-angle pdf at `from` of the direction toward `to`, as an area density at `to`
// (geometric normal ng).
GR_D float to_area(float pdf, V3 from, V3 to, V3 ng) {
    V3 v = to - from;
    float d2 = dot(v, v);
    if (d2 == 0.0f) return 0.0f;
    return pdf * (fabsf(dot(ng, v)) / sqrtf(d2)) / d2;
}

// Stored vertex (BdptVertex, integrators.rs:107-130) as 8 float4, one 128-byte line: the
// shading and connection kernels reach vertices in sorted orders, so a vertex is written
// and read by one thread at a time.
//   0: point, prim     1: incoming, connectible   2: normal, tp.x   3: tangent, tp.y
//   4: binormal, tp.z  5: geom_normal, material   6: emission
//   7: MIS extension: the vertex's MisPart
struct Verts {
    float4* v;
    uint32_t nslots;
    GR_D uint32_t record(uint32_t k, uint32_t slot) const { return k * nslots + slot; }
    GR_D float4& at(uint32_t k, int f, uint32_t slot) const {
        return v[static_cast<size_t>(record(k, slot)) * VREC + f];
    }
};

struct Vtx {
    V3 point, incoming, tp, emission;
    Frame frame;
    uint32_t prim, material;
    bool connectible;
};

GR_D Vtx load_vertex(const Verts& vs, uint32_t k, uint32_t slot) {
    float4 f0 = vs.at(k, 0, slot), f1 = vs.at(k, 1, slot), f2 = vs.at(k, 2, slot), f3 = vs.at(k, 3, slot),
           f4 = vs.at(k, 4, slot), f5 = vs.at(k, 5, slot), f6 = vs.at(k, 6, slot);
    Vtx x;
    x.point = V3{f0.x, f0.y, f0.z};
    x.prim = __float_as_uint(f0.w);
    x.incoming = V3{f1.x, f1.y, f1.z};
    x.connectible = __float_as_uint(f1.w) != 0;
    x.frame.normal = V3{f2.x, f2.y, f2.z};
    x.frame.tangent = V3{f3.x, f3.y, f3.z};
    x.frame.binormal = V3{f4.x, f4.y, f4.z};
    x.frame.geom_normal = V3{f5.x, f5.y, f5.z};
    x.tp = V3{f2.w, f3.w, f4.w};
    x.material = __float_as_uint(f5.w);
    x.emission = V3{f6.x, f6.y, f6.z};
    return x;
}

GR_D void store_vertex(const Verts& vs, uint32_t k, uint32_t slot, V3 point, uint32_t prim, V3 incoming,
                       bool connectible, const Frame& f, V3 tp, uint32_t material, V3 emission) {
    vs.at(k, 0, slot) = make_float4(point.x, point.y, point.z, __uint_as_float(prim));
    vs.at(k, 1, slot) = make_float4(incoming.x, incoming.y, incoming.z, __uint_as_float(connectible ? 1u : 0u));
    vs.at(k, 2, slot) = make_float4(f.normal.x, f.normal.y, f.normal.z, tp.x);
    vs.at(k, 3, slot) = make_float4(f.tangent.x, f.tangent.y, f.tangent.z, tp.y);
    vs.at(k, 4, slot) = make_float4(f.binormal.x, f.binormal.y, f.binormal.z, tp.z);
    vs.at(k, 5, slot) = make_float4(f.geom_normal.x, f.geom_normal.y, f.geom_normal.z, __uint_as_float(material));
    vs.at(k, 6, slot) = make_float4(emission.x, emission.y, emission.z, 0.0f);
}

// Warp-aggregated counter increment for divergent code (the lanes active here).
GR_D uint32_t agg_inc(uint32_t* ctr) {
    unsigned m = __activemask();
    int lane = threadIdx.x & 31;
    int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(ctr, static_cast<uint32_t>(__popc(m)));
    base = __shfl_sync(m, base, leader);
    return base + __popc(m & ((1u << lane) - 1u));
}

GR_D float correct_shading_normal(V3 in_w, V3 out_w, const Frame& f, bool c2l) {  // integrators.rs:232-251
    if (c2l) return 1.0f;
    float num = fabsf(dot(in_w, f.normal)) * fabsf(dot(out_w, f.geom_normal));
    float den = fabsf(dot(in_w, f.geom_normal)) * fabsf(dot(out_w, f.normal));
    if (den == 0.0f) return 0.0f;
    return num / den;
}

GR_D float convert_density(V3 prev, V3 next, const Frame& nf) {  // integrators.rs:253-266
    float dist = magnitude(next - prev);
    if (dist == 0.0f) return 0.0f;
    V3 p2n = (next - prev) / dist;
    return fabsf(dot(nf.normal, p2n)) / (dist * dist);
}

// What a weight needs of a walk for a connection at its vertex n - 1 (n vertices), given the
// connection's own reverse pdfs rev1 and rev2 at vertices n - 1 and n - 2:
//   a = remap0(rev1) / remap0(afwd[n-1]),  b = remap0(rev2) / remap0(afwd[n-2]),
//   part = [cond(n-1)] a^2 + (a b)^2 ([cond(n-2)] + P(n-3)),
// where P(m) = q(m)^2 ([cond(m)] + P(m-1)), q(m) = remap0(arev[m]) / remap0(afwd[m]), sums
// the vertices whose reverse pdfs the connection leaves alone; afwd and arev are the area
// pdfs of a vertex from its predecessor and from its successor.  This is the chained-ratio
// loop (each ratio squared and summed unless the vertex or the one before it is a delta
// vertex) regrouped, so a weight costs O(1).  Everything but rev1 and rev2 depends on the
// walk alone and is known when vertex n - 1 is made: one float4 per vertex.  The camera
// walk's k = 0 term (the light-tracing strategy) is left out where that strategy is.
struct MisPart {
    float fwd1, fwd2;  // remap0(afwd) of vertices n - 1 and n - 2
    float rest;        // [cond(n - 2)] + P(n - 3)
    float cond1;       // [cond(n - 1)]
};
GR_D float remap0(float x) { return x != 0.0f ? x : 1.0f; }
GR_D MisPart load_mis(const Verts& vs, uint32_t k, uint32_t slot) {
    const float4 f7 = vs.at(k, 7, slot);
    return MisPart{f7.x, f7.y, f7.z, f7.w};
}
GR_D void store_mis(const Verts& vs, uint32_t k, uint32_t slot, const MisPart& m) {
    vs.at(k, 7, slot) = make_float4(m.fwd1, m.fwd2, m.rest, m.cond1);
}
GR_D float mis_part(const MisPart& m, uint32_t n, float rev1, float rev2) {
    const float a = remap0(rev1) / m.fwd1;
    float sum = m.cond1 != 0.0f ? a * a : 0.0f;
    if (n >= 2) {
        const float ab = a * (remap0(rev2) / m.fwd2);
        sum += ab * ab * m.rest;
    }
    return sum;
}

// A walk between two vertices.  It travels with its ray in the queue, two float4 per entry
//   (tp.xyz, pdf) (key low, key high, k, flags)
// and with the MIS extension two more
//   (prev.xyz, fwd) (ng.xyz, rest)
// read where the entry sits and written where the surviving walk is pushed.
struct Walk {
    V3 tp;
    float pdf;      // solid-angle pdf of the walk's next direction (0 after a specular sample)
    uint64_t key;
    uint32_t k;     // index of its next vertex
    uint32_t flags; // MIS extension: W_DELTA, W_SKIP0
    V3 prev, ng;    // MIS extension: its last vertex and the geometric normal there
    float fwd;      // remap0(afwd) of its last vertex
    float rest;     // MisPart::rest of its next vertex
};
constexpr uint32_t W_DELTA = 1u;  // the last vertex sampled a specular lobe
constexpr uint32_t W_SKIP0 = 2u;  // camera walk: no light-tracing strategy reaches its first vertex

template <bool MIS>
GR_D Walk load_walk(const float4* __restrict__ q_state, size_t q) {
    const float4* e = q_state + q * (MIS ? 4 : 2);
    const float4 a = e[0], b = e[1];
    Walk w;
    w.tp = V3{a.x, a.y, a.z};
    w.pdf = a.w;
    w.key = (static_cast<uint64_t>(__float_as_uint(b.y)) << 32) | __float_as_uint(b.x);
    w.k = __float_as_uint(b.z);
    w.flags = __float_as_uint(b.w);
    w.prev = w.ng = v3zero();
    w.fwd = w.rest = 0.0f;
    if (MIS) {
        const float4 c = e[2], d = e[3];
        w.prev = V3{c.x, c.y, c.z};
        w.fwd = c.w;
        w.ng = V3{d.x, d.y, d.z};
        w.rest = d.w;
    }
    return w;
}

// Appends this lane's walk and its next ray to a queue with one atomic per warp.  Every lane
// of the warp must call it.
template <bool MIS>
GR_D void push_walk(bool alive, uint32_t* count_out, uint32_t slot, V3 o, V3 d, const Walk& w,
                    uint32_t* __restrict__ nslot, float4* __restrict__ no, float4* __restrict__ nd,
                    float4* __restrict__ nstate, uint32_t cap) {
    const unsigned lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, alive);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == static_cast<unsigned>(leader)) base = atomicAdd(count_out, static_cast<uint32_t>(__popc(m)));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (alive) {
        const uint32_t pos = base + __popc(m & ((1u << lane) - 1u));
        if (!GR_IN_RANGE(pos, cap)) return;
        nslot[pos] = slot;
        no[pos] = make_float4(o.x, o.y, o.z, 0.0f);
        nd[pos] = make_float4(d.x, d.y, d.z, 0.0f);
        float4* e = nstate + static_cast<size_t>(pos) * (MIS ? 4 : 2);
        e[0] = make_float4(w.tp.x, w.tp.y, w.tp.z, w.pdf);
        e[1] = make_float4(__uint_as_float(static_cast<uint32_t>(w.key)),
                           __uint_as_float(static_cast<uint32_t>(w.key >> 32)), __uint_as_float(w.k),
                           __uint_as_float(w.flags));
        if (MIS) {
            e[2] = make_float4(w.prev.x, w.prev.y, w.prev.z, w.fwd);
            e[3] = make_float4(w.ng.x, w.ng.y, w.ng.z, w.rest);
        }
    }
}

// Per path: vertex counts of both walks, flags and the throughput at the camera walk's
// escape (with F_ESCAPE).
struct PathOut {
    uint32_t* vcount;
    uint32_t* flags;
    float4* escape;
};

template <bool MIS>
__global__ void __launch_bounds__(BLOCK) k_bdpt_raygen(DeviceScene s, BdptParams p, Verts vs, PathOut out,
                                                       float2* __restrict__ st_buf, uint32_t* count_out,
                                                       uint32_t* __restrict__ nslot, float4* __restrict__ no,
                                                       float4* __restrict__ nd, float4* __restrict__ nstate) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool cam_alive = false, light_alive = false;
    V3 co = v3zero(), cd = v3zero(), lo = v3zero(), ld = v3zero();
    Walk cw{}, lw{};
    if (i < p.n) {
        const PathSample ps = path_sample(p.order, i);
        uint64_t key = path_key(p.seed, p.first_pass + ps.pass, ps.row * p.width + ps.col);
        float s0, t0;
        film_sample_point(p.width, p.height, ps.row, ps.col, key, s0, t0);
        camera_ray(p.cam, s0, t0, co, cd);
        st_buf[ps.slot] = make_float2(s0, t0);
        uint32_t fl = 0, light_vertices = 0;
        cw.tp = v3one();
        cw.pdf = MIS ? p.view.dir_pdf(dot(cd, -p.view.axis[2])) : 0.0f;
        cw.key = lw.key = key;
        cw.prev = p.view.pos;
        cam_alive = p.max_len > 0;
        if (s.num_lights > 0) {
            float u[6];
            for (int k = 0; k < 6; ++k) u[k] = uniform01(key, DIM_LIGHT_SAMPLE + k);
            DevLightSample ls = sample_light(s, u);
            if (ls.point_pdf == 0.0f || ls.dir_pdf == 0.0f) {
                fl |= F_SKIP;
            } else {
                uint32_t mi = __ldg(s.prim_material + ls.prim);
                const DevMaterial& m = s.materials[mi];
                V3 ie = light_world(m, ls.direction, ls.frame) *
                        (fabsf(dot(ls.frame.geom_normal, ls.direction)) / (ls.point_pdf * ls.dir_pdf));
                store_vertex(vs, 0, 2 * i + 1, ls.origin, ls.prim, v3zero(), true, ls.frame, v3one() / ls.point_pdf,
                             mi, v3zero());
                light_vertices = 1;
                lw.tp = ie;
                lw.pdf = ls.dir_pdf;
                lw.k = 1;
                if (MIS) {
                    lw.fwd = remap0(ls.point_pdf);
                    store_mis(vs, 0, 2 * i + 1, MisPart{lw.fwd, 1.0f, 0.0f, 1.0f});
                    lw.prev = ls.origin;
                    lw.ng = ls.frame.geom_normal;
                    lw.rest = 1.0f;
                }
                light_alive = !is_zero(ie) && 1 < p.max_len;
                lo = nudge(ls.origin, ls.direction);
                ld = ls.direction;
            }
        }
        out.vcount[2 * i] = 0;
        out.vcount[2 * i + 1] = light_vertices;
        out.flags[i] = fl;
    }
    push_walk<MIS>(cam_alive, count_out, 2 * i, co, cd, cw, nslot, no, nd, nstate, p.nslots);
    push_walk<MIS>(light_alive, count_out, 2 * i + 1, lo, ld, lw, nslot, no, nd, nstate, p.nslots);
}

// One vertex of random_walk (integrators.rs:138-229) at the hit h = (t, leaf-order primitive
// or -1, u, v) of walk `slot`'s ray (o, d): stores the vertex and advances w.  Returns
// whether the walk goes on, with its next ray; a walk that ends leaves its vertex count.
// `lobe`: the lobe that shade_bucket picked.
template <bool MIS>
GR_D bool walk_vertex(const DeviceScene& s, const BdptParams& p, const Verts& vs, const PathOut& out, uint32_t slot,
                      Walk& w, uint32_t lobe, V3 o, V3 d, float4 h, V3& new_o, V3& new_d) {
    const uint32_t walk = slot & 1u, path = slot >> 1, k = w.k;
    if (!GR_IN_RANGE(k, p.max_len) || !GR_IN_RANGE(slot, p.nslots)) return false;
    const bool c2l = walk == 0;
    const int32_t pk = __float_as_int(h.y);
    if (pk < 0) {
        // As if a black infinite light was hit (integrators.rs:210-225).  Such a vertex
        // connects to nothing and every term with it is zero, so it is not stored or
        // counted.  The throughput at the escape is kept for the environment extension.
        if (walk == 0) {
            out.escape[path] = make_float4(w.tp.x, w.tp.y, w.tp.z, 0.0f);
            out.flags[path] |= F_ESCAPE;
        }
        out.vcount[slot] = k;
        return false;
    }
    uint32_t prim;
    Frame f = hit_frame(s, pk, o, d, h.x, h.z, h.w, prim);
    uint32_t mi = __ldg(s.prim_material + prim);
    const DevMaterial& m = s.materials[mi];
    uint32_t base = (walk ? DIM_LIGHT_WALK : DIM_CAMERA_WALK) + 4 * k;
    V3 incoming = -d;
    V3 hit_point = o + (d * h.x);
    MaterialSample ms = sample_lobe(m, incoming, f, c2l, static_cast<int>(lobe), uniform01(w.key, base + 1),
                                    uniform01(w.key, base + 2));
    bool connectible = count_lobes(m, LOBE_DIFFUSE | LOBE_GLOSSY) != 0;
    V3 ntp = mul(w.tp, ms.radiance * (fabsf(dot(f.normal, ms.outgoing)) / ms.pdf));
    ntp = ntp * correct_shading_normal(incoming, ms.outgoing, f, c2l);
    store_vertex(vs, k, slot, hit_point, prim, incoming, connectible, f, w.tp, mi, ms.emission);
    const bool delta = (ms.kind & LOBE_SPECULAR) != 0;
    if (MIS) {
        // Area pdf of this vertex from its predecessor, and of the predecessor from this
        // vertex (reverse BSDF pdf; zero after a specular sample, PBRT 3e section 16.3.2).
        MisPart part;
        part.fwd1 = remap0(to_area(w.pdf, w.prev, hit_point, f.geom_normal));
        float P = 0.0f;  // P(k - 1), which the next vertex's part needs
        if (k == 0) {  // of a camera walk
            float ss, tt, dd, cv;
            if (!(p.lt && p.view.project(hit_point, ss, tt, dd, cv))) w.flags |= W_SKIP0;
            part.fwd2 = 1.0f;
            part.rest = 0.0f;
            part.cond1 = w.flags & W_SKIP0 ? 0.0f : 1.0f;
        } else {
            part.fwd2 = w.fwd;
            part.rest = w.rest;
            part.cond1 = w.flags & W_DELTA ? 0.0f : 1.0f;
            const float rev = delta ? 0.0f : pdf_world(m, ms.outgoing, incoming, f);
            const float q = remap0(to_area(rev, hit_point, w.prev, w.ng)) / w.fwd;
            P = q * q * w.rest;
        }
        store_mis(vs, k, slot, part);
        const bool before_delta = k >= 1 && (w.flags & W_DELTA);
        const bool cond = !delta && !before_delta && !(k == 0 && (w.flags & W_SKIP0));
        w.rest = (cond ? 1.0f : 0.0f) + P;
        w.fwd = part.fwd1;
        w.prev = hit_point;
        w.ng = f.geom_normal;
        w.flags = (w.flags & ~W_DELTA) | (delta ? W_DELTA : 0u);
    }
    if (k + 1 >= p.rr_len || nearly_zero(ntp)) {
        float rv = uniform01(w.key, base + 3);
        float prob = clamped_lerp(0.25f, 0.75f, luminance(ntp));
        ntp = rv < prob ? ntp / prob : v3zero();
    }
    const bool alive = !is_zero(ntp) && k + 1 < p.max_len;
    new_o = nudge(hit_point, ms.outgoing);
    new_d = ms.outgoing;
    w.tp = ntp;
    w.pdf = delta ? 0.0f : ms.pdf;
    w.k = k + 1;
    if (!alive) out.vcount[slot] = k + 1;
    return alive;
}

// BDPT walk shading in blocks of GR_BDPT_SHADE_BLOCK threads (128 or 768), each sorting its
// chunk by code path; at 768 one block fills an SM (85 registers), so its warps shade the
// same code path at a time (as the path tracer's k_shade, where 768 measured 9% faster).
#ifndef GR_BDPT_SHADE_BLOCK
#define GR_BDPT_SHADE_BLOCK 768
#endif
constexpr int BSBLOCK = GR_BDPT_SHADE_BLOCK;
static_assert(BSBLOCK == 128 || BSBLOCK == 768, "BDPT shading block of 128 or 768 threads");
constexpr uint32_t BSHADE_PER_THREAD = BSBLOCK == 128 ? SHADE_PER_THREAD : SHADE_ONE_CHUNK;

template <bool MIS>
__global__ void __launch_bounds__(BSBLOCK, 768 / BSBLOCK)
    k_bdpt_shade(DeviceScene s, BdptParams p, Verts vs, PathOut out, const uint32_t* __restrict__ count_in,
                 const uint32_t* __restrict__ q_slot, const float4* __restrict__ q_o, const float4* __restrict__ q_d,
                 const float4* __restrict__ q_hit, const float4* __restrict__ q_state, uint32_t* count_out,
                 uint32_t* __restrict__ nslot, float4* __restrict__ no, float4* __restrict__ nd,
                 float4* __restrict__ nstate) {
    extern __shared__ unsigned char dsmem[];
    const SortView sm = sort_view<BSBLOCK, BSHADE_PER_THREAD>(dsmem);
    const uint32_t n = *count_in;
    // Material-sorted shading (shade_sort.cuh), by (walk, material, chosen lobe).
    // Block-uniform chunk loop.
    const uint32_t per =
        chunk_per_thread<BSBLOCK, BSBLOCK == 128 ? BSHADE_PER_THREAD : SHADE_BIG_PER, BSHADE_PER_THREAD>(n, gridDim.x);
    const uint32_t chunk = chunk_entries<BSBLOCK>(n, gridDim.x, per);
    for (uint32_t c0 = blockIdx.x * chunk; c0 < n; c0 += gridDim.x * chunk) {
        const uint32_t cn = min(chunk, n - c0);
        sort_chunk<BSBLOCK, BSHADE_PER_THREAD>(sm, cn, per, [&](uint32_t i) {
            const uint32_t q = c0 + i;
            const uint32_t w = q_slot[q] & 1u;
            const float4 b = q_state[static_cast<size_t>(q) * (MIS ? 4 : 2) + 1];
            const uint64_t key = (static_cast<uint64_t>(__float_as_uint(b.y)) << 32) | __float_as_uint(b.x);
            const uint32_t dim = (w ? DIM_LIGHT_WALK : DIM_CAMERA_WALK) + 4 * __float_as_uint(b.z);
            return shade_bucket(s, __float_as_int(q_hit[q].y), uniform01(key, dim), w);
        });
        for (uint32_t e = 0; e < per; ++e) {
            uint32_t i = e * BSBLOCK + threadIdx.x;
            bool alive = false;
            uint32_t slot = 0;
            V3 new_o = v3zero(), new_d = v3zero();
            Walk w{};
            if (i < cn) {
                const uint32_t at = sm.order[i];
                uint32_t q = c0 + at;
                slot = q_slot[q];
                const float4 o4 = q_o[q], d4 = q_d[q];
                w = load_walk<MIS>(q_state, q);
                alive = walk_vertex<MIS>(s, p, vs, out, slot, w, sorted_lobe(sm, at), V3{o4.x, o4.y, o4.z},
                                         V3{d4.x, d4.y, d4.z}, q_hit[q], new_o, new_d);
            }
            push_walk<MIS>(alive, count_out, slot, new_o, new_d, w, nslot, no, nd, nstate, p.nslots);
        }
        __syncthreads();  // sm is reused by the next chunk
    }
}

// A walk in the path loop; without the MIS extension its second half stays behind.
struct LoopWalk {
    uint32_t slot, unused;
    Walk w;
};
static_assert(sizeof(Walk) == 64, "its first half is the walk without the MIS extension");
template <bool MIS>
constexpr int loop_words() {
    return MIS ? 18 : 10;
}

// Carries a queue's walks to their end (run_paths).
template <int W, bool MIS>
__global__ void __launch_bounds__(PATH_LOOP_THREADS, PATH_LOOP_BLOCKS)
    k_bdpt_walks(DeviceScene s, BdptParams p, Verts vs, PathOut out, const uint32_t* __restrict__ count,
                 const uint32_t* __restrict__ q_slot, const float4* __restrict__ q_o, const float4* __restrict__ q_d,
                 const float4* __restrict__ q_state, uint32_t* fetch, int* err, unsigned long long* rays) {
    extern __shared__ unsigned char smem[];
    int2 spill[MAX_STACK - SMEM_STACK];
    const auto stk = thread_stack<PATH_LOOP_THREADS>(smem, spill);
    const uint32_t n = *count;
    if (n == 0) return;
    auto take = [&](uint32_t q, LoopWalk& path, V3& o, V3& d) {
        path.slot = q_slot[q];
        path.unused = 0;
        const float4 o4 = q_o[q], d4 = q_d[q];
        o = V3{o4.x, o4.y, o4.z};
        d = V3{d4.x, d4.y, d4.z};
        path.w = load_walk<MIS>(q_state, q);
    };
    auto bucket = [&](const LoopWalk& path, int32_t k) {
        const uint32_t walk = path.slot & 1u;
        const uint32_t dim = (walk ? DIM_LIGHT_WALK : DIM_CAMERA_WALK) + 4 * path.w.k;
        return shade_bucket(s, k, uniform01(path.w.key, dim), walk);
    };
    auto shade = [&](LoopWalk& path, uint32_t lobe, V3 o, V3 d, float4 h, V3& no, V3& nd) {
        return walk_vertex<MIS>(s, p, vs, out, path.slot, path.w, lobe, o, d, h, no, nd);
    };
    count_rays(run_paths<W, loop_words<MIS>(), LoopWalk>(
                   stk, smem, n, fetch, err, err + 1, s.num_components >= GROUPED_COMPONENTS,
                   [&]() -> const DeviceScene& { return s; }, take, bucket, shade),
               rays);
}

// Capacities of the strategy entries and of the shadow queue, as BdptState::ensure sizes
// them (checked builds test every write against them).
[[maybe_unused]] GR_D size_t entry_cap(const BdptParams& p) { return static_cast<size_t>(p.n) * (p.max_len * (p.max_len + 1) / 2); }
[[maybe_unused]] GR_D size_t shadow_cap(const BdptParams& p) { return entry_cap(p) + (p.lt ? static_cast<size_t>(p.n) * p.max_len : 0); }

// ---------------------------------------------------- MIS extension (power heuristic)
// Veach 1997 eq. 10.9 with beta = 2, in the ratio form of PBRT 3e section 16.3.4: per
// vertex the area pdfs of generating it along its own walk (afwd) and from the other
// side (arev), ratios of neighbouring strategies' pdfs chained outwards from the
// connection, delta (specular) vertices skipped and zero pdfs counted as 1.  The
// strategies are (c camera-walk, l light-walk vertices), c + l <= max_len, and with
// light tracing also c = 0.  The oracle states the same weight as a loop over the
// strategies (orender.hpp, mis_weight); MisPart regroups it.

// Area pdf with which Bvh::sample_light picks a point of light prim `prim`
// (bvh.rs:481-496, mesh.rs:310-327, sphere.rs:103-111).
GR_D float light_point_pdf(const DeviceScene& s, uint32_t prim) {
    for (uint32_t k = 0; k < s.num_lights; ++k) {
        const LightRec& L = s.lights[k];
        if (L.prim != prim) continue;
        float pdf = L.type == PRIM_SPHERE ? 1.0f / (4.0f * PI * L.radius * L.radius) : 1.0f / L.area;
        return pdf / static_cast<float>(s.num_lights);
    }
    return 0.0f;
}

// Pdf of a light emitting toward w: cosine about the geometric normal (prim.rs:37-51).
GR_D float light_dir_pdf(const Frame& f, V3 w) {
    float c = dot(f.geom_normal, w);
    return c > 0.0f ? c * FRAC_1_PI : 0.0f;
}

struct VPos {
    V3 point, ng;
};
GR_D VPos load_pos(const Verts& vs, uint32_t k, uint32_t slot) {
    float4 f0 = vs.at(k, 0, slot), f5 = vs.at(k, 5, slot);
    return VPos{V3{f0.x, f0.y, f0.z}, V3{f5.x, f5.y, f5.z}};
}

// A walk vertex's BSDF toward a connection: the value f(wi, wo) (material.rs:66-93) and,
// for the MIS weights, pdf(wi, wo) and pdf(wo, wi) (material.rs:95-119), each summed in
// the same order as f_world / pdf_world.  One out-of-line copy serves every call site of
// the connection kernel, whose divergent warps otherwise miss in the instruction cache
// on many inlined copies of the Disney mixture.
struct VEval {
    V3 f;
    float pdf_fwd, pdf_rev;
};
static __device__ __noinline__ VEval eval_vertex(const DevMaterial& m, V3 wi, V3 wo, const Frame& fr, bool c2l,
                                                 bool pdfs) {
    VEval e{v3zero(), 0.0f, 0.0f};
    V3 il = world_to_local(wi, fr.tangent, fr.binormal, fr.normal);
    V3 ol = world_to_local(wo, fr.tangent, fr.binormal, fr.normal);
    bool refl = (dot(wi, fr.geom_normal) * dot(wo, fr.geom_normal)) > 0.0f;
    float pf = 0.0f, pr = 0.0f;
#pragma unroll 1
    for (int k = 0; k < m.n_lobes; ++k) {
        const DevLobe& L = m.lobe[k];
        const bool value = (refl && (L.kind & LOBE_REFLECTION)) || (!refl && (L.kind & LOBE_TRANSMISSION));
        const LobeEval v = lobe_eval(L, il, ol, c2l, (value ? WANT_F : 0u) | (pdfs ? WANT_PDF | WANT_REV : 0u));
        if (value) e.f = e.f + v.f;
        pf += v.pdf;
        pr += v.rev;
    }
    if (pdfs && m.n_lobes) {
        const float n = static_cast<float>(m.n_lobes);
        e.pdf_fwd = il.z == 0.0f ? 0.0f : pf / n;
        e.pdf_rev = ol.z == 0.0f ? 0.0f : pr / n;
    }
    return e;
}

// MIS weight of camera strategy (c >= 1, l >= 0) with a non-zero connection.  For l >= 1, ez and ey are the connection's evaluations at
// z (camera side, toward y) and y (light side, toward z; for l = 1 the light's
// direction pdf in pdf_fwd).
GR_D float strategy_weight(const DeviceScene& s, const Verts& vs, uint32_t i, uint32_t c, uint32_t l, const Vtx& z,
                           const Vtx* y, const VEval& ez, const VEval& ey) {
    float z_rev = 0.0f, zm_rev = 0.0f, y_rev = 0.0f, ym_rev = 0.0f;
    if (l == 0) {  // the camera walk hit a light
        z_rev = light_point_pdf(s, z.prim);
        if (c >= 2) {
            VPos zp = load_pos(vs, c - 2, 2 * i);
            zm_rev = to_area(light_dir_pdf(z.frame, z.incoming), z.point, zp.point, zp.ng);
        }
    } else {
        z_rev = to_area(ey.pdf_fwd, y->point, z.point, z.frame.geom_normal);
        if (c >= 2) {
            VPos zp = load_pos(vs, c - 2, 2 * i);
            zm_rev = to_area(ez.pdf_rev, z.point, zp.point, zp.ng);
        }
        y_rev = to_area(ez.pdf_fwd, z.point, y->point, y->frame.geom_normal);
        if (l >= 2) {
            VPos yp = load_pos(vs, l - 2, 2 * i + 1);
            ym_rev = to_area(ey.pdf_rev, y->point, yp.point, yp.ng);
        }
    }
    const float camera_part = mis_part(load_mis(vs, c - 1, 2 * i), c, z_rev, zm_rev);
    const float light_part = l ? mis_part(load_mis(vs, l - 1, 2 * i + 1), l, y_rev, ym_rev) : 0.0f;
    return 1.0f / (1.0f + camera_part + light_part);
}

// ------------------------------------------------ connection items: paths by strategy
// Paths are counting-sorted by their (camera, light) vertex counts (17 x 17 buckets, walks
// <= 16), so the paths with cs camera vertices and at least l light vertices are
// consecutive: from start[17 cs + l] to start[17 (cs + 1)].  The strategies of all paths
// are items: item t belongs to a segment (l, c, cs), the paths of exactly cs camera and at
// least l light vertices doing strategy (c, l), and is the (t - base)-th of that range.
// Segments of one l and c follow each other, so a warp evaluates one strategy of 32 paths:
// one connection each, instead of one path each with its own loops over both walks.
// Light-tracing items are segments (l, cs) in the same way.  Which thread handles which
// path changes no result.
constexpr uint32_t LENS = 17;
constexpr uint32_t LEN_BUCKETS = LENS * LENS;
constexpr uint32_t MAX_SEGMENTS = 1496;    // sum over c of (17 - c)^2, walks <= 16
constexpr uint32_t MAX_LT_SEGMENTS = 272;  // 16 x 17

struct Items {
    uint32_t hist[LEN_BUCKETS];       // paths per bucket, then next free position
    uint32_t start[LEN_BUCKETS + 1];  // first position of each bucket
    uint32_t segments, lt_segments;
    uint32_t base[MAX_SEGMENTS + 1];  // first item per segment, then the number of items
    uint32_t what[MAX_SEGMENTS];      // (l << 16) | (c << 8) | cs
    uint32_t at[LENS * LENS * LENS];  // base of segment (l, c, cs)
    uint32_t lt_base[MAX_LT_SEGMENTS + 1];
    uint32_t lt_what[MAX_LT_SEGMENTS];  // (l << 8) | cs
};

GR_D uint32_t len_bucket(const uint32_t* vcount, const uint32_t* flags, uint32_t i) {
    if (flags[i] & F_SKIP) return 0;
    return min(vcount[2 * i], 16u) * LENS + min(vcount[2 * i + 1], 16u);
}

__global__ void __launch_bounds__(BLOCK) k_bdpt_len_count(uint32_t n, const uint32_t* __restrict__ vcount,
                                                          const uint32_t* __restrict__ flags, Items* items) {
    __shared__ uint32_t h[LEN_BUCKETS];
    for (uint32_t b = threadIdx.x; b < LEN_BUCKETS; b += blockDim.x) h[b] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&h[len_bucket(vcount, flags, i)], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < LEN_BUCKETS; b += blockDim.x)
        if (h[b]) atomicAdd(&items->hist[b], h[b]);
}

// Exclusive prefix sum of one value per thread of a PLAN_THREADS-thread block; `total`
// gets the sum.
constexpr uint32_t PLAN_THREADS = 512;
GR_D uint32_t block_scan(uint32_t* sm, uint32_t v, uint32_t& total) {
    const uint32_t t = threadIdx.x;
    __syncthreads();  // sm is free
    sm[t] = v;
    __syncthreads();
    for (uint32_t o = 1; o < PLAN_THREADS; o <<= 1) {
        const uint32_t x = t >= o ? sm[t - o] : 0u;
        __syncthreads();
        sm[t] += x;
        __syncthreads();
    }
    total = sm[PLAN_THREADS - 1];
    return sm[t] - v;
}

// One block: bucket counts -> first positions, and the segments of the items.
__global__ void __launch_bounds__(PLAN_THREADS) k_bdpt_items(Items* items, uint32_t max_len, uint32_t lt) {
    __shared__ uint32_t sm[PLAN_THREADS], start[LEN_BUCKETS + 1];
    const uint32_t t = threadIdx.x;
    static_assert(LEN_BUCKETS < PLAN_THREADS, "one bucket per thread");
    uint32_t total;
    const uint32_t first = block_scan(sm, t < LEN_BUCKETS ? items->hist[t] : 0u, total);
    if (t < LEN_BUCKETS) {
        start[t] = first;
        items->hist[t] = first;
        items->start[t] = first;
    }
    if (t == 0) {
        start[LEN_BUCKETS] = total;
        items->start[LEN_BUCKETS] = total;
    }
    __syncthreads();
    auto paths = [&](uint32_t cs, uint32_t l) { return start[(cs + 1) * LENS] - start[cs * LENS + l]; };
    // Segments in the order l, c, cs, each thread a run of PER of them.
    constexpr uint32_t PER = (MAX_SEGMENTS + PLAN_THREADS - 1) / PLAN_THREADS;
    uint32_t what[PER], size[PER], mine = 0, count = 0;
    for (uint32_t k = 0; k < PER; ++k) what[k] = size[k] = 0;
    for (uint32_t l = 0; l < max_len; ++l)
        for (uint32_t c = 1; c + l <= max_len; ++c) {
            const uint32_t n = max_len - c + 1;  // cs = c .. max_len
            for (uint32_t k = 0; k < PER; ++k) {
                const uint32_t g = t * PER + k;
                if (g >= count && g < count + n) {
                    const uint32_t cs = c + (g - count);
                    what[k] = (l << 16) | (c << 8) | cs;
                    size[k] = paths(cs, l);
                    mine += size[k];
                }
            }
            count += n;
        }
    uint32_t base = block_scan(sm, mine, total);
    for (uint32_t k = 0; k < PER; ++k) {
        const uint32_t g = t * PER + k;
        if (g >= count) break;
        items->what[g] = what[k];
        items->base[g] = base;
        items->at[((what[k] >> 16) * LENS + ((what[k] >> 8) & 255u)) * LENS + (what[k] & 255u)] = base;
        base += size[k];
    }
    if (t == 0) {
        items->segments = count;
        items->base[count] = total;
    }
    // Light-tracing segments: l = 1 .. max_len, cs = 0 .. max_len (a camera walk that
    // escapes at once has no vertex).
    const uint32_t lt_count = lt ? max_len * (max_len + 1) : 0u;
    const uint32_t l = t / (max_len + 1) + 1, cs = t % (max_len + 1);
    const uint32_t n = t < lt_count ? paths(cs, l) : 0u;
    base = block_scan(sm, n, total);
    if (t < lt_count) {
        items->lt_what[t] = (l << 8) | cs;
        items->lt_base[t] = base;
    }
    if (t == 0) {
        items->lt_segments = lt_count;
        items->lt_base[lt_count] = total;
    }
}

__global__ void __launch_bounds__(BLOCK) k_bdpt_len_scatter(uint32_t n, const uint32_t* __restrict__ vcount,
                                                            const uint32_t* __restrict__ flags, Items* items,
                                                            uint32_t* __restrict__ order) {
    const unsigned lane = threadIdx.x & 31u;
    for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
        const uint32_t i = b + threadIdx.x;
        const bool in = i < n;
        const uint32_t key = in ? len_bucket(vcount, flags, i) : 0xFFFFFFFFu;
        // One atomic per distinct bucket in the warp.
        const unsigned same = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(same) - 1;
        uint32_t base = 0;
        if (in && static_cast<int>(lane) == leader)
            base = atomicAdd(&items->hist[key], static_cast<uint32_t>(__popc(same)));
        base = __shfl_sync(0xffffffffu, base, leader);
        const uint32_t at = base + __popc(same & ((1u << lane) - 1u));
        if (in && GR_IN_RANGE(at, n)) order[at] = i;
    }
}

// The segment of item t: the last one whose base is <= t (empty segments share their base
// with the next, which is then taken).
GR_D uint32_t find_segment(const uint32_t* base, uint32_t segments, uint32_t t) {
    uint32_t lo = 0, hi = segments;
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (base[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

// One strategy of one path per thread: connect() without its visibility test, times the
// strategy's weight (uniform or MIS), into entries[t]; terms that need the test queue a
// shadow ray.
// Bound by divergence (the two materials of a connection differ within a warp) and by the
// instruction fetch of the mixture.  512 x 512 x 16 spp with MIS: one thread per path,
// looping over its strategies, 4.94 ms; items 3.54 (with field-major vertices replaced by
// whole lines), without the escapes' vertices 1.62.  Cornell box, 200 x 150 x 4 spp, length
// 16: 841 -> 164 us.  Sorting chunks of items by the two materials' lobes cost as much as
// it saved; 3 / 4 / 5 blocks per SM measured the same (9.58 / 9.60 / 9.55 ms per render; 4 has no spills).
#ifndef GR_CONNECT_BLOCK
#define GR_CONNECT_BLOCK 128
#endif
#ifndef GR_CONNECT_MIN_BLOCKS
#define GR_CONNECT_MIN_BLOCKS 4
#endif
__global__ void __launch_bounds__(GR_CONNECT_BLOCK, GR_CONNECT_MIN_BLOCKS)
    k_bdpt_connect(DeviceScene s, BdptParams p, Verts vs, const Items* __restrict__ items,
                   const uint32_t* __restrict__ order, uint32_t* counters, float4* __restrict__ entries,
                   uint4* __restrict__ shadow_q) {
    __shared__ uint32_t base[MAX_SEGMENTS + 1];
    const uint32_t segments = items->segments;
    for (uint32_t k = threadIdx.x; k <= segments; k += blockDim.x) base[k] = items->base[k];
    __syncthreads();
    const uint32_t total = base[segments];
    const uint32_t extra = p.lt ? 1u : 0u;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t g = find_segment(base, segments, t);
        const uint32_t what = __ldg(&items->what[g]);
        const uint32_t l = what >> 16, c = (what >> 8) & 255u, cs = what & 255u;
        const uint32_t i = order[__ldg(&items->start[cs * LENS + l]) + (t - base[g])];
        V3 term = v3zero();
        float flag = E_NO_TEST;
        const Vtx cv = load_vertex(vs, c - 1, 2 * i);
        Vtx lv;
        VEval ez{v3zero(), 0.0f, 0.0f}, ey{v3zero(), 0.0f, 0.0f};
        if (l == 0) {
            term = mul(cv.tp, cv.emission);
        } else if (cv.connectible) {
            lv = load_vertex(vs, l - 1, 2 * i + 1);
            if (lv.connectible) {
                V3 c2l = normalized(lv.point - cv.point);
                V3 l2c = -c2l;  // equals normalized(cv.point - lv.point) bit for bit
                const DevMaterial& cm = s.materials[cv.material];
                const DevMaterial& lm = s.materials[lv.material];
                ez = eval_vertex(cm, cv.incoming, c2l, cv.frame, true, p.mis);
                V3 cr = ez.f;
                V3 ce;
                if (l == 1) {
                    ce = light_world(lm, l2c, lv.frame);
                    ey.pdf_fwd = light_dir_pdf(lv.frame, l2c);
                } else {
                    ey = eval_vertex(lm, lv.incoming, l2c, lv.frame, false, p.mis);
                    ce = ey.f;
                }
                float gcos = fabsf(dot(cv.frame.normal, c2l));
                float cdn = convert_density(cv.point, lv.point, lv.frame);
                term = mul(mul(mul(cv.tp, cr), ce), lv.tp) * (gcos * cdn);
                if (!nearly_zero(term)) {
                    flag = E_PENDING;
                    uint32_t sq = agg_inc(counters + CNT_SHADOWQ);
                    if (GR_IN_RANGE(sq, shadow_cap(p)))  // the two vertices' records
                        shadow_q[sq] = make_uint4(t, vs.record(c - 1, 2 * i), vs.record(l - 1, 2 * i + 1), 0);
                }
            }
        }
        float w;
        if (!p.mis) w = 1.0f / static_cast<float>(c + l + extra);  // integrators.rs:345-354
        else w = is_zero(term) ? 0.0f : strategy_weight(s, vs, i, c, l, cv, l ? &lv : nullptr, ez, ey);
        term = term * w;
        if (GR_IN_RANGE(t, entry_cap(p))) entries[t] = make_float4(term.x, term.y, term.z, flag);
    }
}

// The light-tracing strategy (t = 1, an MIS extension), one light-walk vertex per thread:
// inside the image it gets a camera term in lt[t] (value, flag) and its film pixel in
// lt_pixel[t].
__global__ void __launch_bounds__(BLOCK) k_bdpt_light_trace(DeviceScene s, BdptParams p, Verts vs,
                                                            const Items* __restrict__ items,
                                                            const uint32_t* __restrict__ order, uint32_t* counters,
                                                            uint4* __restrict__ shadow_q, float4* __restrict__ lt,
                                                            uint32_t* __restrict__ lt_pixel) {
    __shared__ uint32_t base[MAX_LT_SEGMENTS + 1];
    const uint32_t segments = items->lt_segments;
    for (uint32_t k = threadIdx.x; k <= segments; k += blockDim.x) base[k] = items->lt_base[k];
    __syncthreads();
    const uint32_t total = base[segments];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t g = find_segment(base, segments, t);
        const uint32_t what = __ldg(&items->lt_what[g]);
        const uint32_t l = what >> 8, cs = what & 255u;
        const uint32_t i = order[__ldg(&items->start[cs * LENS + l]) + (t - base[g])];
        // Light-walk vertex y -> camera.  We / pdf of a pinhole camera is
        // 1 / (area cos^3 dist^2) (PBRT 3e section 16.1.1).
        float4 out = make_float4(0.0f, 0.0f, 0.0f, E_NO_TEST);
        uint32_t pix = 0;
        const Vtx y = load_vertex(vs, l - 1, 2 * i + 1);
        float ss, tt, dist, cvw;
        if (y.connectible && p.view.project(y.point, ss, tt, dist, cvw)) {
            V3 w_yc = (p.view.pos - y.point) / dist;
            const DevMaterial& ym = s.materials[y.material];
            VEval ev{v3zero(), 0.0f, 0.0f};
            if (l >= 2) ev = eval_vertex(ym, y.incoming, w_yc, y.frame, false, p.mis);
            V3 F = l == 1 ? light_world(ym, w_yc, y.frame) : ev.f;
            float gcos = fabsf(dot(y.frame.normal, w_yc)) / (p.view.area * cvw * cvw * cvw * dist * dist);
            V3 L = mul(y.tp, F) * gcos;
            if (!nearly_zero(L)) {
                float w;
                if (!p.mis) {
                    w = 1.0f / static_cast<float>(l + 1);
                } else {
                    float y_rev = to_area(p.view.dir_pdf(cvw), p.view.pos, y.point, y.frame.geom_normal);
                    float ym_rev = 0.0f;
                    if (l >= 2) {
                        VPos yp = load_pos(vs, l - 2, 2 * i + 1);
                        ym_rev = to_area(ev.pdf_rev, y.point, yp.point, yp.ng);
                    }
                    w = 1.0f / (1.0f + mis_part(load_mis(vs, l - 1, 2 * i + 1), l, y_rev, ym_rev));
                }
                L = L * w;
                uint32_t col = min(p.width - 1, static_cast<uint32_t>(floorf(0.5f * (ss + 1.0f) * p.width)));
                uint32_t row = min(p.height - 1, static_cast<uint32_t>(floorf(0.5f * (tt + 1.0f) * p.height)));
                pix = row * p.width + col;
                out = make_float4(L.x, L.y, L.z, E_PENDING);
                uint32_t sq = agg_inc(counters + CNT_SHADOWQ);
                if (GR_IN_RANGE(sq, shadow_cap(p))) shadow_q[sq] = make_uint4(t, vs.record(l - 1, 2 * i + 1), 0, 1);
            }
        }
        if (GR_IN_RANGE(t, static_cast<size_t>(p.n) * p.max_len)) {
            lt[t] = out;
            lt_pixel[t] = pix;
        }
    }
}

// Shadow query entries: (entry, record of vertex a, of vertex b, kind).  Kind 0 connects
// two walk vertices (their strategy entry); kind 1 connects the camera to vertex a (a
// light-tracing entry in lt).
template <int W>
__global__ void __launch_bounds__(BLOCK) k_bdpt_shadow(DeviceScene s, uint32_t* counters,
                                                       const uint4* __restrict__ shadow_q, const float4* __restrict__ v0,
                                                       float4* __restrict__ entries, float4* __restrict__ lt,
                                                       float3 cam, int* err, unsigned long long* shadow_rays) {
    extern __shared__ unsigned char smem[];
    int2 spill[MAX_STACK - SMEM_STACK];
    const auto stk = thread_stack<BLOCK>(smem, spill);
    const uint32_t n = counters[CNT_SHADOWQ];
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(shadow_rays, static_cast<unsigned long long>(n));
    uint4 e = make_uint4(0, 0, 0, 0);
    auto answer = [&](bool visible) { (e.w == 1 ? lt : entries)[e.x].w = visible ? E_VISIBLE : E_OCCLUDED; };
    trace_queue<W, true, false>(
        n, stk, err, nullptr, nullptr, SharedCounter{counters + CNT_SHADOWF}, [&]() -> const DeviceScene& { return s; },
        [&](uint32_t q, TravState& t) {
            e = shadow_q[q];
            V3 a, b;
            if (e.w == 1) {  // Bvh::visibility(camera, y), as the oracle's light-tracing test
                float4 y4 = v0[static_cast<size_t>(e.y) * VREC];
                a = V3{cam.x, cam.y, cam.z};
                b = V3{y4.x, y4.y, y4.z};
            } else {
                float4 a4 = v0[static_cast<size_t>(e.y) * VREC], b4 = v0[static_cast<size_t>(e.z) * VREC];
                a = V3{a4.x, a4.y, a4.z};
                b = V3{b4.x, b4.y, b4.z};
            }
            if (fabsf(a.x - b.x) < 1e-3f && fabsf(a.y - b.y) < 1e-3f && fabsf(a.z - b.z) < 1e-3f) {
                answer(false);
                return false;
            }
            const V3 d = normalized(b - a);
            const V3 o = nudge(a, d);
            trav_init(t, o, d, magnitude(b - o) - 1e-3f);
            return true;
        },
        [&](uint32_t, const TravState& t) { answer(t.hit < 0); });
}

// Sums each path's weighted strategy terms in loop order.  Threads take the paths in the
// items' order, so the entries of one strategy are read consecutively.
__global__ void __launch_bounds__(BLOCK) k_bdpt_gather(DeviceScene s, BdptParams p,
                                                       const uint32_t* __restrict__ vcount,
                                                       const uint32_t* __restrict__ flags,
                                                       const float4* __restrict__ escape,
                                                       const Items* __restrict__ items,
                                                       const uint32_t* __restrict__ order,
                                                       const float4* __restrict__ entries, float4* __restrict__ L_out) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= p.n) return;
    const uint32_t i = order[t];
    const uint32_t fl = flags[i];
    V3 light = v3zero();
    if (s.has_env && (fl & F_ESCAPE)) {
        float4 e = escape[i];
        light = light + mul(V3{e.x, e.y, e.z}, V3{s.env[0], s.env[1], s.env[2]});
    }
    if (!(fl & F_SKIP)) {
        const uint32_t cs = vcount[2 * i], ls = vcount[2 * i + 1];
        for (uint32_t c = 1; c <= cs; ++c) {
            for (uint32_t l = 0; l <= ls && c + l <= p.max_len; ++l) {
                const uint32_t at = __ldg(&items->at[(l * LENS + c) * LENS + cs]);
                const float4 e = entries[at + (t - __ldg(&items->start[cs * LENS + l]))];
                V3 term = (e.w == E_NO_TEST || e.w == E_VISIBLE) ? V3{e.x, e.y, e.z} : v3zero();
                light = light + term;  // weighted in k_bdpt_connect
            }
        }
    }
    L_out[path_sample(p.order, i).slot] = make_float4(light.x, light.y, light.z, 0.0f);
}

// Adds the visible light-tracing terms to the film's splat buffer.
__global__ void __launch_bounds__(BLOCK) k_bdpt_splat(const Items* __restrict__ items, const float4* __restrict__ lt,
                                                      const uint32_t* __restrict__ lt_pixel, float4* splat) {
    const uint32_t total = items->lt_base[items->lt_segments];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const float4 v = lt[t];
        if (v.w != E_VISIBLE) continue;
        float* d = reinterpret_cast<float*>(splat + lt_pixel[t]);
        atomicAdd(d, v.x);
        atomicAdd(d + 1, v.y);
        atomicAdd(d + 2, v.z);
    }
}

__global__ void k_bdpt_samples_out(uint32_t n, const float2* __restrict__ st, const float4* __restrict__ L,
                                   float* out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[5 * i] = st[i].x;
    out[5 * i + 1] = st[i].y;
    out[5 * i + 2] = L[i].x;
    out[5 * i + 3] = L[i].y;
    out[5 * i + 4] = L[i].z;
}

uint32_t max_pairs(uint32_t max_len) { return max_len * (max_len + 1) / 2; }

template <int W>
gr_status shadow_launch(const DeviceScene& s, uint32_t cap, uint32_t* counters, const uint4* q, const float4* v0,
                        float4* entries, float4* lt, float3 cam, int* err, unsigned long long* shadow_rays,
                        cudaStream_t st) {
    size_t smem = step_stack_smem_bytes(BLOCK);
    int grid = resident_grid(k_bdpt_shadow<W>, smem, cap);
    k_bdpt_shadow<W><<<grid, BLOCK, smem, st>>>(s, counters, q, v0, entries, lt, cam, err, shadow_rays);
    GR_CUDA_TRY(cudaGetLastError());
    return GR_OK;
}

template <int W, bool MIS>
gr_status walks_launch(const DeviceScene& s, const BdptParams& p, const Verts& vs, const PathOut& out, uint32_t most,
                       BdptState& bs, int cur, uint32_t* cnt, int* err, unsigned long long* rays, cudaStream_t st) {
    const size_t smem = path_loop_smem_bytes(loop_words<MIS>());
    int grid;
    GR_TRY_S(path_loop_grid(k_bdpt_walks<W, MIS>, smem, most, grid));
    k_bdpt_walks<W, MIS><<<grid, PATH_LOOP_THREADS, smem, st>>>(
        s, p, vs, out, cnt + CNT_LOOP, bs.q_slot[cur].as<uint32_t>(), bs.q_o[cur].as<float4>(),
        bs.q_d[cur].as<float4>(), bs.q_state[cur].as<float4>(), cnt + CNT_LOOP_FETCH, err, rays);
    GR_CUDA_TRY(cudaGetLastError());
    return GR_OK;
}

// Both walks of a group's paths: raygen, then bounce by bounce; once at most PATH_LOOP_MAX
// walks are left, one launch carries them to their
// end: Cornell box, 200 x 150 x 4 spp, length 16, 636 us of extension and shading -> 404.
template <bool MIS>
gr_status run_walks(const DeviceScene& s, const BdptParams& p, const Verts& vs, BdptState& bs, uint32_t* cnt, int* err,
                    unsigned long long* rays, uint64_t& launches, cudaStream_t st) {
    const PathOut out{bs.vcount.as<uint32_t>(), bs.flags.as<uint32_t>(), bs.escape.as<float4>()};
    BounceReadback& rb = device_work().readback;  // the caller holds device_work().mu
    GR_CUDA_TRY(rb.ensure());
    k_bdpt_raygen<MIS><<<(p.n + BLOCK - 1) / BLOCK, BLOCK, 0, st>>>(
        s, p, vs, out, bs.st.as<float2>(), cnt + CNT_QUEUE0, bs.q_slot[0].as<uint32_t>(), bs.q_o[0].as<float4>(),
        bs.q_d[0].as<float4>(), bs.q_state[0].as<float4>());
    GR_CUDA_TRY(cudaGetLastError());
    ++launches;
    QueueOutlook look(p.nslots);
    // Every walk ends within max_len bounces (one vertex per bounce).
    for (uint32_t depth = 0; depth < p.max_len; ++depth) {
        const int cur = depth & 1, nxt = cur ^ 1;
        const bool loop = look.offer();
        GR_TRY_S(bounce_begin(rb, cnt, depth, loop ? PATH_LOOP_MAX : 0u, st));
        if (loop) {
            const uint32_t most = std::min(look.bound, PATH_LOOP_MAX);
            switch (s.width) {
                case 2: GR_TRY_S((walks_launch<2, MIS>(s, p, vs, out, most, bs, cur, cnt, err, rays, st))); break;
                case 4: GR_TRY_S((walks_launch<4, MIS>(s, p, vs, out, most, bs, cur, cnt, err, rays, st))); break;
                default: GR_TRY_S((walks_launch<8, MIS>(s, p, vs, out, most, bs, cur, cnt, err, rays, st)));
            }
            ++launches;
            if (look.bound <= PATH_LOOP_MAX) break;  // the path loop takes it whatever its length
        }
        GR_TRY_S(extend_any(s, false, look.bound, cnt + cur, bs.q_o[cur].as<float4>(), bs.q_d[cur].as<float4>(),
                            bs.q_hit.as<float4>(), err, rays, cnt + CNT_FETCH, st, false));
        GR_CUDA_TRY(cudaGetLastError());
        const size_t ssmem = sort_smem_bytes(BSBLOCK, BSHADE_PER_THREAD);
        GR_CUDA_TRY(allow_sort_smem(k_bdpt_shade<MIS>, ssmem));
        k_bdpt_shade<MIS><<<resident_grid(k_bdpt_shade<MIS>, ssmem, look.bound, BSBLOCK), BSBLOCK, ssmem, st>>>(
            s, p, vs, out, cnt + cur, bs.q_slot[cur].as<uint32_t>(), bs.q_o[cur].as<float4>(),
            bs.q_d[cur].as<float4>(), bs.q_hit.as<float4>(), bs.q_state[cur].as<float4>(), cnt + nxt,
            bs.q_slot[nxt].as<uint32_t>(), bs.q_o[nxt].as<float4>(), bs.q_d[nxt].as<float4>(),
            bs.q_state[nxt].as<float4>());
        GR_CUDA_TRY(cudaGetLastError());
        launches += 2;
        bool more = true;
        GR_TRY_S(bounce_wait(rb, depth, look, more));
        if (!more) break;
    }
    return GR_OK;
}

}  // namespace

size_t BdptState::bytes_per_path(uint32_t max_len) {
    const size_t pairs = max_pairs(max_len);
    return 2 * (2 * (4 + 16 + 16 + 64) + 16) + 8 + 16      // queues (with state), hits; st, light
           + 2 * max_len * VREC * 16 + 2 * 4 + 4 + 16         // vertices, counts, flags, escape
           + pairs * 16 + (pairs + max_len) * 16 + max_len * (16 + 4) + 4;  // entries, shadow queue, lt, order
}

cudaError_t BdptState::ensure(size_t paths, uint32_t max_len) {
    size_t slots = 2 * paths;
    size_t pairs = static_cast<size_t>(max_pairs(max_len)) * paths;
    cudaError_t e;
    for (int k = 0; k < 2; ++k) {
        if ((e = q_slot[k].ensure(slots * sizeof(uint32_t))) != cudaSuccess) return e;
        if ((e = q_o[k].ensure(slots * sizeof(float4))) != cudaSuccess) return e;
        if ((e = q_d[k].ensure(slots * sizeof(float4))) != cudaSuccess) return e;
        if ((e = q_state[k].ensure(slots * 4 * sizeof(float4))) != cudaSuccess) return e;
    }
    if ((e = q_hit.ensure(slots * sizeof(float4))) != cudaSuccess) return e;
    if ((e = st.ensure(paths * sizeof(float2))) != cudaSuccess) return e;
    if ((e = light.ensure(paths * sizeof(float4))) != cudaSuccess) return e;
    if ((e = verts.ensure(slots * max_len * VREC * sizeof(float4))) != cudaSuccess) return e;
    if ((e = vcount.ensure(slots * sizeof(uint32_t))) != cudaSuccess) return e;
    if ((e = flags.ensure(paths * sizeof(uint32_t))) != cudaSuccess) return e;
    if ((e = escape.ensure(paths * sizeof(float4))) != cudaSuccess) return e;
    if ((e = entries.ensure(pairs * sizeof(float4))) != cudaSuccess) return e;
    const size_t lt_n = paths * max_len;  // light-tracing terms
    if ((e = shadow.ensure((pairs + lt_n) * sizeof(uint4))) != cudaSuccess) return e;
    if ((e = lt.ensure(lt_n * sizeof(float4))) != cudaSuccess) return e;
    if ((e = lt_pixel.ensure(lt_n * sizeof(uint32_t))) != cudaSuccess) return e;
    if ((e = order.ensure(paths * sizeof(uint32_t))) != cudaSuccess) return e;
    if ((e = items.ensure(sizeof(Items))) != cudaSuccess) return e;
    return cudaSuccess;
}

gr_status render_bdpt(gr_scene* sc, const RenderJob& job, cudaStream_t st) {
    const gr_render_params& rp = job.params;
    const uint32_t npix = job.width * job.height;
    const uint32_t total = job.samples_out ? 1u : rp.spp;
    if (total == 0) return GR_OK;
    const uint32_t max_len = rp.max_depth ? rp.max_depth : 16;
    // Paths in flight: up to 4 M (the bench's 512x512 x 16 spp in one group; 0.5 M -> 1 M
    // -> 2 M -> 4 M measured 96 -> 117 -> 135 -> 146 Msamples/s with MIS), within the
    // smaller of 24 GB and a quarter of free device memory.
    const char* env = std::getenv("GR_BDPT_PATHS_IN_FLIGHT");
    uint32_t target;
    if (env && std::atoi(env) > 0) {
        target = static_cast<uint32_t>(std::atoi(env));
    } else {
        size_t free_b = 0, total_b = 0;
        GR_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
        const size_t budget = std::min<size_t>(size_t(24) << 30, free_b / 4);
        const size_t fit = budget / BdptState::bytes_per_path(max_len);
        target = static_cast<uint32_t>(std::max<size_t>(1u << 19, std::min<size_t>(1u << 22, fit)));
    }
    uint32_t group = std::max(1u, std::min(total, target / std::max(1u, npix)));
    const size_t npaths = static_cast<size_t>(group) * npix;
    BdptState& bs = device_work().bdpt;
    GR_CUDA_TRY(bs.ensure(npaths, max_len));
    BdptState& ps = bs;
    uint32_t* cnt = sc->counters.as<uint32_t>();
    int* err = reinterpret_cast<int*>(cnt + CNT_ERROR);
    unsigned long long* rays = reinterpret_cast<unsigned long long*>(cnt + CNT_RAYS);
    unsigned long long* shadow = reinterpret_cast<unsigned long long*>(cnt + CNT_SHADOW);
    uint64_t launches = 0;

    BdptParams p;
    p.cam = job.camera;
    p.width = job.width;
    p.height = job.height;
    p.seed = rp.seed;
    p.max_len = max_len;
    p.rr_len = rp.rr_depth;
    p.mis = rp.mis ? 1u : 0u;
    p.lt = rp.light_tracing ? 1u : 0u;
    {  // the camera seen from the scene (rotation rows and translation of the camera matrix)
        const DevCamera& c = job.camera;
        p.view.pos = V3{c.m[3][0] / c.m[3][3], c.m[3][1] / c.m[3][3], c.m[3][2] / c.m[3][3]};
        for (int k = 0; k < 3; ++k) p.view.axis[k] = V3{c.m[k][0], c.m[k][1], c.m[k][2]};
        p.view.wx = c.wx;
        p.view.wy = c.wy;
        p.view.area = 4.0f * c.wx * c.wy;
    }
    const float3 cam_pos = make_float3(p.view.pos.x, p.view.pos.y, p.view.pos.z);
    for (uint32_t done = 0; done < total; done += group) {
        uint32_t g = std::min(group, total - done);
        p.n = g * npix;
        p.nslots = 2 * p.n;
        p.first_pass = rp.first_pass + done;
        Verts vs{bs.verts.as<float4>(), p.nslots};
        GR_CUDA_TRY(cudaMemsetAsync(cnt + CNT_QUEUE0, 0, sizeof(uint32_t), st));
        GR_CUDA_TRY(cudaMemsetAsync(cnt + CNT_SHADOWQ, 0, 2 * sizeof(uint32_t), st));
        p.order = make_path_order(job.width, job.height, g);
        GR_TRY_S(p.mis || p.lt ? run_walks<true>(job.scene, p, vs, bs, cnt, err, rays, launches, st)
                               : run_walks<false>(job.scene, p, vs, bs, cnt, err, rays, launches, st));
        Items* items = bs.items.as<Items>();
        {
            const int sgrid = static_cast<int>(std::min<uint32_t>((p.n + BLOCK - 1) / BLOCK, 1024u));
            GR_CUDA_TRY(cudaMemsetAsync(items->hist, 0, sizeof(items->hist), st));
            k_bdpt_len_count<<<sgrid, BLOCK, 0, st>>>(p.n, bs.vcount.as<uint32_t>(), bs.flags.as<uint32_t>(), items);
            k_bdpt_items<<<1, PLAN_THREADS, 0, st>>>(items, max_len, p.lt);
            k_bdpt_len_scatter<<<sgrid, BLOCK, 0, st>>>(p.n, bs.vcount.as<uint32_t>(), bs.flags.as<uint32_t>(), items,
                                                       bs.order.as<uint32_t>());
            GR_CUDA_TRY(cudaGetLastError());
            launches += 3;
        }
        // The number of items is known on the device only: every resident block, looping.
        const uint32_t all = p.n * max_pairs(max_len);
        k_bdpt_connect<<<resident_grid(k_bdpt_connect, 0, all, GR_CONNECT_BLOCK), GR_CONNECT_BLOCK, 0, st>>>(
            job.scene, p, vs, items, bs.order.as<uint32_t>(), cnt, bs.entries.as<float4>(), bs.shadow.as<uint4>());
        GR_CUDA_TRY(cudaGetLastError());
        if (p.lt) {
            k_bdpt_light_trace<<<resident_grid(k_bdpt_light_trace, 0, p.n * max_len), BLOCK, 0, st>>>(
                job.scene, p, vs, items, bs.order.as<uint32_t>(), cnt, bs.shadow.as<uint4>(), bs.lt.as<float4>(),
                bs.lt_pixel.as<uint32_t>());
            GR_CUDA_TRY(cudaGetLastError());
            ++launches;
        }
        uint32_t cap = p.n * (max_pairs(max_len) + (p.lt ? max_len : 0u));
        gr_status s2;
        switch (job.scene.width) {
            case 2: s2 = shadow_launch<2>(job.scene, cap, cnt, bs.shadow.as<uint4>(), bs.verts.as<float4>(),
                                          bs.entries.as<float4>(), bs.lt.as<float4>(), cam_pos, err, shadow, st); break;
            case 4: s2 = shadow_launch<4>(job.scene, cap, cnt, bs.shadow.as<uint4>(), bs.verts.as<float4>(),
                                          bs.entries.as<float4>(), bs.lt.as<float4>(), cam_pos, err, shadow, st); break;
            default: s2 = shadow_launch<8>(job.scene, cap, cnt, bs.shadow.as<uint4>(), bs.verts.as<float4>(),
                                           bs.entries.as<float4>(), bs.lt.as<float4>(), cam_pos, err, shadow, st); break;
        }
        if (s2 != GR_OK) return s2;
        k_bdpt_gather<<<(p.n + BLOCK - 1) / BLOCK, BLOCK, 0, st>>>(
            job.scene, p, bs.vcount.as<uint32_t>(), bs.flags.as<uint32_t>(), bs.escape.as<float4>(), items,
            bs.order.as<uint32_t>(), bs.entries.as<float4>(), ps.light.as<float4>());
        GR_CUDA_TRY(cudaGetLastError());
        if (p.lt && job.splat) {
            k_bdpt_splat<<<resident_grid(k_bdpt_splat, 0, p.n * max_len), BLOCK, 0, st>>>(
                items, bs.lt.as<float4>(), bs.lt_pixel.as<uint32_t>(), job.splat);
            GR_CUDA_TRY(cudaGetLastError());
            ++launches;
        }
        launches += 3;
        if (job.film) {
            DevBuf& fs = device_work().film_sched;
            GR_CUDA_TRY(fs.ensure(film_sched_words(job.width, job.height) * sizeof(uint32_t)));
            gr_status s3 = film_gather(ps.st.as<float2>(), ps.light.as<float4>(), job.width, job.height, g, job.film,
                                       st, fs.as<uint32_t>(), err);
            if (s3 != GR_OK) return s3;
            ++launches;
        }
        if (job.samples_out) {
            k_bdpt_samples_out<<<(p.n + 255) / 256, 256, 0, st>>>(p.n, ps.st.as<float2>(), ps.light.as<float4>(),
                                                                 job.samples_out);
            GR_CUDA_TRY(cudaGetLastError());
            ++launches;
        }
    }
    sc->stats.samples += static_cast<uint64_t>(total) * npix;
    sc->stats.kernel_launches += launches;
    return GR_OK;
}

gr_status bdpt_index_check() {
#if GR_CHECKED
    bool bad = false;
    GR_CUDA_TRY(take_bad_index(bad));
    if (bad) {
        set_error("BDPT: a queue or entry index was out of range (checked build)");
        return GR_ERR_INTERNAL;
    }
#endif
    return GR_OK;
}

}  // namespace gr
