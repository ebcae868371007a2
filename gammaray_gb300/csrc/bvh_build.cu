// Device BVH builds: a binary tree made on the GPU, then collapsed into the same wide node
// layout as the host build, so traversal is unchanged.  GR_BUILD_DEVICE_LBVH makes a linear
// BVH, as follows; the reference's SAH tree of large scenes is sah_build.cuh's.
//
//   records    boxes and primitive records from the caller's vertex and index arrays, with
//              the index checks (large scenes of few prims; else the host makes them)
//   bounds     centroid bounds of all components (block reduction + ordered-int atomics)
//   morton     30-bit Morton code of each centroid in those bounds
//   sort       codes with component indices (CUB radix sort, stable: equal codes keep
//              component order)
//   tree       binary radix tree over the sorted codes (Karras, "Maximizing parallelism
//              in the construction of BVHs, octrees, and k-d trees", HPG 2012): internal
//              node i finds its key range and split from common-prefix lengths; equal
//              codes are told apart by their sorted index
//   boxes      bottom-up: each leaf walks to the root; the second child to arrive at a
//              node computes its box (counter atomics, no waiting)
//   collapse   level by level from the root, with no host step in between: a wide node
//              takes its binary node's two children and opens the largest-area child
//              holding more than `leaf_size` components until it has `width` children; a
//              child of at most `leaf_size` components becomes one leaf over its
//              contiguous range.  Going down it also finds the exact worst-case traversal
//              stack use (the host collapse's: the largest sum of children - 1 along a path)
//   permute    primitive records and attribute indices into leaf order
//
// The linear tree differs from the reference's SAH tree; closest hits do not (a ray keeps the
// nearest hit over all primitives), except that a tie at exactly equal distance may go
// to the other primitive.
#include <algorithm>
#include <cfloat>
#include <memory>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "runtime.hpp"
#include "traverse.cuh"  // MAX_STACK, the traversal stack bound

namespace gr {

namespace {

constexpr int BB = 256;  // threads per block of the build kernels

// Float <-> int that orders like the float, for atomicMin / atomicMax.
GR_D int ordered(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
GR_D float unordered(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

// Centroid = 0.5 lo + 0.5 hi (bvh.rs:26).
GR_D V3 centroid(const float* __restrict__ box, uint32_t k) {
    const float* b = box + 6 * static_cast<size_t>(k);
    return V3{0.5f * b[0] + 0.5f * b[3], 0.5f * b[1] + 0.5f * b[4], 0.5f * b[2] + 0.5f * b[5]};
}

__global__ void k_centroid_bounds(const float* __restrict__ box, uint32_t n, int* bounds) {
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        V3 c = centroid(box, k);
        float v[3] = {c.x, c.y, c.z};
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], v[a]);
            hi[a] = fmaxf(hi[a], v[a]);
        }
    }
    for (int a = 0; a < 3; ++a)
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    __shared__ int sb[6];  // of the block: one atomic per bound and block reaches memory
    if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? 0x7FFFFFFF : static_cast<int>(0x80000000u);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        for (int a = 0; a < 3; ++a) {
            atomicMin(sb + a, ordered(lo[a]));
            atomicMax(sb + 3 + a, ordered(hi[a]));
        }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(bounds + threadIdx.x, sb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(bounds + threadIdx.x, sb[threadIdx.x]);
}

// Spreads the low 10 bits of v to every third bit.
GR_D uint32_t spread3(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void k_morton(const float* __restrict__ box, uint32_t n, const int* __restrict__ bounds,
                         uint32_t* __restrict__ code, uint32_t* __restrict__ index) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    V3 c = centroid(box, k);
    float v[3] = {c.x, c.y, c.z};
    uint32_t q[3];
    for (int a = 0; a < 3; ++a) {
        float lo = unordered(bounds[a]), hi = unordered(bounds[3 + a]);
        float ext = hi - lo;
        float t = ext > 0.0f ? (v[a] - lo) / ext : 0.5f;
        t = fminf(fmaxf(t, 0.0f), 1.0f);
        q[a] = min(1023u, static_cast<uint32_t>(t * 1024.0f));
    }
    code[k] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    index[k] = k;
}

// Common-prefix length of sorted keys i and j (codes, then sorted indices); -1 out of range.
GR_D int delta(const uint32_t* __restrict__ code, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint32_t a = code[i], b = code[j];
    if (a == b) return 32 + __clz(static_cast<uint32_t>(i ^ j));
    return __clz(a ^ b);
}

// Child references: >= 0 an internal node, < 0 the leaf (sorted component) ~ref.
// split[i]: both child references and both component counts of internal node i.
__global__ void k_radix_tree(const uint32_t* __restrict__ code, int n, int4* __restrict__ split,
                             int* __restrict__ parent_internal, int* __restrict__ parent_leaf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = delta(code, n, i, i + 1) - delta(code, n, i, i - 1) >= 0 ? 1 : -1;
    const int dmin = delta(code, n, i, i - d);
    int lmax = 2;
    while (delta(code, n, i, i + lmax * d) > dmin) lmax <<= 1;  // at most log2(n) + 1 doublings
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(code, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(code, n, i, j);
    int s = 0;
    for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
        if (delta(code, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = lo == gamma ? ~gamma : gamma;
    const int right = hi == gamma + 1 ? ~(gamma + 1) : gamma + 1;
    split[i] = make_int4(left, right, gamma - lo + 1, hi - gamma);
    if (left >= 0) parent_internal[left] = i;
    else parent_leaf[~left] = i;
    if (right >= 0) parent_internal[right] = i;
    else parent_leaf[~right] = i;
}

struct NodeBox {
    float lo[3], hi[3];
};

GR_D NodeBox leaf_box(const float* __restrict__ box, const uint32_t* __restrict__ perm, int k) {
    const float* b = box + 6 * static_cast<size_t>(perm[k]);
    return NodeBox{{b[0], b[1], b[2]}, {b[3], b[4], b[5]}};
}

// An internal node as the collapse opens it: both children's boxes, references and counts.
struct alignas(16) Opened {
    float4 l0, l1, r0, r1;  // (lo.xyz, ref) (hi.xyz, count) of the left and of the right child
};

// The box of an internal node, from its children's, written by another thread (past L1).
GR_D NodeBox load_node_box(const Opened* nodes, int i) {
    const float4* f = reinterpret_cast<const float4*>(nodes + i);
    const float4 l0 = __ldcg(f), l1 = __ldcg(f + 1), r0 = __ldcg(f + 2), r1 = __ldcg(f + 3);
    return NodeBox{{fminf(l0.x, r0.x), fminf(l0.y, r0.y), fminf(l0.z, r0.z)},
                   {fmaxf(l1.x, r1.x), fmaxf(l1.y, r1.y), fmaxf(l1.z, r1.z)}};
}

__global__ void k_boxes(const float* __restrict__ box, const uint32_t* __restrict__ perm, int n,
                        const int4* __restrict__ split, const int* __restrict__ parent_internal,
                        const int* __restrict__ parent_leaf, Opened* nodes, int* visits, int* err) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int p = parent_leaf[k];
    for (int steps = 0; p >= 0; ++steps) {
        if (steps >= n) {  // a parent chain longer than the tree: flag it, never loop
            atomicExch(err, 1);
            return;
        }
        __threadfence();  // this child's boxes are visible before the count
        if (atomicAdd(visits + p, 1) == 0) return;  // the sibling will finish the node
        const int4 c = split[p];
        const NodeBox a = c.x < 0 ? leaf_box(box, perm, ~c.x) : load_node_box(nodes, c.x);
        const NodeBox b = c.y < 0 ? leaf_box(box, perm, ~c.y) : load_node_box(nodes, c.y);
        Opened o;
        o.l0 = make_float4(a.lo[0], a.lo[1], a.lo[2], __int_as_float(c.x));
        o.l1 = make_float4(a.hi[0], a.hi[1], a.hi[2], __int_as_float(c.z));
        o.r0 = make_float4(b.lo[0], b.lo[1], b.lo[2], __int_as_float(c.y));
        o.r1 = make_float4(b.hi[0], b.hi[1], b.hi[2], __int_as_float(c.w));
        nodes[p] = o;
        p = parent_internal[p];
    }
}

// A child of a wide node: its binary node (>= 0) or leaf ~k, its component range and box.
struct Cand {
    int ref, first, count;
    float area;  // half its surface area; -1 when it is not to be opened
    NodeBox box;
};

GR_D float half_area(const NodeBox& b) {
    float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return dx * dy + dy * dz + dz * dx;
}

GR_D Cand cand_of(const float4 c0, const float4 c1, int first) {
    Cand c;
    c.ref = __float_as_int(c0.w);
    c.first = first;
    c.count = __float_as_int(c1.w);
    c.box = NodeBox{{c0.x, c0.y, c0.z}, {c1.x, c1.y, c1.z}};
    c.area = half_area(c.box);
    return c;
}

// Levels of the wide tree.  The linear tree is at most 30 (code bits) + 32 (index bits of
// equal codes) deep, so its collapse has no more.  A SAH tree can be deeper: one whose
// collapse is goes to the host build.
constexpr uint32_t MAX_LEVELS = 64;

struct CollapseCtl {
    uint32_t count[MAX_LEVELS + 1];  // wide nodes per level, numbered level by level
    uint32_t stack;                  // largest stack use along a path so far
};

// The wide nodes of one level: node w stands for binary node todo[w].x (the root leaf: -1),
// todo[w].y is its first component, .z its component count and .w the stack entries its
// ancestors may hold.  The level's size is read on the device, so levels follow each other
// without the host.
template <int W>
__global__ void __launch_bounds__(BB) k_collapse(CollapseCtl* ctl, const int* __restrict__ err, uint32_t level,
                                                 int4* __restrict__ todo,
                                                 const Opened* __restrict__ opened, const float* __restrict__ box,
                                                 const uint32_t* __restrict__ perm, uint32_t leaf_size,
                                                 float* __restrict__ nodes, [[maybe_unused]] uint32_t room) {
    const uint32_t n = ctl->count[level];
    if (n == 0 || *err) return;  // (a flagged tree is not walked)
    uint32_t begin = 0;
    for (uint32_t l = 0; l < level; ++l) begin += ctl->count[l];
    const unsigned lane = threadIdx.x & 31u;
    uint32_t deepest = 0;
    // Warp-uniform trip counts: every lane reaches the shuffles.
    for (uint32_t f0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; f0 < n; f0 += gridDim.x * blockDim.x) {
        const bool in = f0 + lane < n;
        const uint32_t wide = begin + f0 + lane;
        Cand c[W];
        int nc = 0;
        uint32_t inner = 0, held = 0;
        if (in) {
            const int4 job = todo[wide];
            held = static_cast<uint32_t>(job.w);
            auto open = [&](int ref, int first, Cand& l, Cand& r) {
                const Opened o = opened[ref];
                l = cand_of(o.l0, o.l1, first);
                r = cand_of(o.r0, o.r1, first + l.count);
            };
            if (job.x >= 0 && job.z > static_cast<int>(leaf_size)) {
                open(job.x, job.y, c[0], c[1]);
                nc = 2;
            } else {  // a scene of one leaf
                c[0].ref = job.x;
                c[0].first = job.y;
                c[0].count = job.z;
                c[0].area = -1.0f;
                c[0].box = leaf_box(box, perm, job.y);
                for (int k = 1; k < job.z; ++k) {
                    const NodeBox b = leaf_box(box, perm, job.y + k);
                    for (int a = 0; a < 3; ++a) {
                        c[0].box.lo[a] = fminf(c[0].box.lo[a], b.lo[a]);
                        c[0].box.hi[a] = fmaxf(c[0].box.hi[a], b.hi[a]);
                    }
                }
                nc = 1;
            }
            while (nc < W) {  // open the largest-area child that is still too big for a leaf
                int best = -1;
                float best_area = -1.0f;
                for (int q = 0; q < nc; ++q) {
                    if (c[q].ref < 0 || c[q].count <= static_cast<int>(leaf_size)) continue;
                    if (!(c[q].area <= best_area)) {
                        best = q;
                        best_area = c[q].area;
                    }
                }
                if (best < 0) break;
                const int ref = c[best].ref, first = c[best].first;
                for (int q = nc; q > best + 1; --q) c[q] = c[q - 1];
                open(ref, first, c[best], c[best + 1]);
                ++nc;
            }
            for (int j = 0; j < nc; ++j) inner += c[j].count > static_cast<int>(leaf_size) ? 1u : 0u;
        }
        // Numbers of the next level's nodes: one atomic per warp.
        uint32_t before = inner;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= static_cast<unsigned>(o)) before += x;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, before, 31);
        uint32_t base = 0;
        if (lane == 0 && total) base = atomicAdd(&ctl->count[level + 1], total);
        uint32_t next = begin + n + __shfl_sync(0xffffffffu, base, 0) + before - inner;
        if (!in) continue;
        held += static_cast<uint32_t>(nc - 1);
        deepest = max(deepest, held);
        float* node = nodes + static_cast<size_t>(wide) * 8 * W;
        for (int j = 0; j < W; ++j) {
            NodeBox b{{FLT_MAX, FLT_MAX, FLT_MAX}, {-FLT_MAX, -FLT_MAX, -FLT_MAX}};  // empty slots never hit
            int ref = ~0;
            if (j < nc) {
                b = c[j].box;
                if (c[j].count <= static_cast<int>(leaf_size)) {
                    ref = ~static_cast<int>((static_cast<uint32_t>(c[j].first) << LEAF_COUNT_BITS) |
                                            static_cast<uint32_t>(c[j].count - 1));
                } else {
                    ref = static_cast<int>(next);
                    if (GR_IN_RANGE(next, room)) todo[next] = make_int4(c[j].ref, c[j].first, c[j].count, static_cast<int>(held));
                    ++next;
                }
            }
            for (int a = 0; a < 3; ++a) {
                node[a * W + j] = b.lo[a];
                node[(3 + a) * W + j] = b.hi[a];
            }
            node[6 * W + j] = __int_as_float(ref);
        }
        for (int j = 6 * W + W; j < 8 * W; ++j) node[j] = 0.0f;
    }
    deepest = __reduce_max_sync(0xffffffffu, deepest);
    if (lane == 0 && deepest) atomicMax(&ctl->stack, deepest);
}

// A prim's part of the caller's arrays, on the device.
struct PrimSrc {
    uint32_t first;  // its first component
    uint32_t sphere, num_vertices, num_normals, num_uvs;
    uint32_t nbase, ubase;  // its attributes in the scene's arrays
    const float* vertices;
    const uint32_t *tris, *tri_normals, *tri_uvs;
    float center[3], radius;
};

constexpr int ERR_BAD_INDEX = 2;  // k_records: a triangle's index is out of range

// Component k: its box, its primitive record (the host's put_record) and its attribute
// indices; out-of-range indices are flagged and read nothing.
__global__ void k_records(const PrimSrc* __restrict__ prims, uint32_t num_prims, uint32_t n, float* __restrict__ box,
                          float4* __restrict__ rec, uint32_t* __restrict__ tn, uint32_t* __restrict__ tu, int* err) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t p = 0;
    for (uint32_t hi = num_prims; hi - p > 1;) {  // the last prim whose first component is <= k
        const uint32_t mid = p + (hi - p) / 2;
        if (prims[mid].first <= k) p = mid;
        else hi = mid;
    }
    const PrimSrc& s = prims[p];
    const uint32_t t = k - s.first;
    float lo[3], hi[3];
    float4 r0, r1, r2;
    if (s.sphere) {
        for (int a = 0; a < 3; ++a) {  // Sphere::bbox_world (sphere.rs:47-58)
            lo[a] = s.center[a] - s.radius;
            hi[a] = s.center[a] + s.radius;
        }
        r0 = make_float4(s.center[0], s.center[1], s.center[2], __uint_as_float(p));
        r1 = make_float4(s.radius, 0.0f, 0.0f, __uint_as_float(0u));
        r2 = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(PRIM_SPHERE));
        for (int q = 0; q < 3; ++q) {
            if (tn) tn[3 * static_cast<size_t>(k) + q] = NO_INDEX;
            if (tu) tu[3 * static_cast<size_t>(k) + q] = NO_INDEX;
        }
    } else {
        uint32_t v[3], nn[3] = {NO_INDEX, NO_INDEX, NO_INDEX}, uu[3] = {NO_INDEX, NO_INDEX, NO_INDEX};
        bool bad = false;
        for (int q = 0; q < 3; ++q) {
            v[q] = s.tris[3 * static_cast<size_t>(t) + q];
            bad |= v[q] >= s.num_vertices;
        }
        if (s.tri_normals && s.tri_normals[3 * static_cast<size_t>(t)] != NO_INDEX)
            for (int q = 0; q < 3; ++q) {
                const uint32_t i = s.tri_normals[3 * static_cast<size_t>(t) + q];
                bad |= i >= s.num_normals;
                nn[q] = s.nbase + i;
            }
        if (s.tri_uvs)
            for (int q = 0; q < 3; ++q) {
                const uint32_t i = s.tri_uvs[3 * static_cast<size_t>(t) + q];
                bad |= i >= s.num_uvs;
                uu[q] = s.ubase + i;
            }
        if (bad) {
            atomicExch(err, ERR_BAD_INDEX);
            v[0] = v[1] = v[2] = 0;  // a mesh has vertices (checked on the host)
        }
        float c[3][3];
        for (int q = 0; q < 3; ++q)
            for (int a = 0; a < 3; ++a) c[q][a] = bad ? 0.0f : s.vertices[3 * static_cast<size_t>(v[q]) + a];
        for (int a = 0; a < 3; ++a) {  // Mesh::bbox_world (mesh.rs:262-268)
            lo[a] = fminf(fminf(fminf(FLT_MAX, c[0][a]), c[1][a]), c[2][a]);
            hi[a] = fmaxf(fmaxf(fmaxf(-FLT_MAX, c[0][a]), c[1][a]), c[2][a]);
        }
        // c, a - c and b - c (mesh.rs:278)
        r0 = make_float4(c[2][0], c[2][1], c[2][2], __uint_as_float(p));
        r1 = make_float4(c[0][0] - c[2][0], c[0][1] - c[2][1], c[0][2] - c[2][2], __uint_as_float(t));
        r2 = make_float4(c[1][0] - c[2][0], c[1][1] - c[2][1], c[1][2] - c[2][2], __int_as_float(PRIM_TRIANGLE));
        for (int q = 0; q < 3; ++q) {
            if (tn) tn[3 * static_cast<size_t>(k) + q] = nn[q];
            if (tu) tu[3 * static_cast<size_t>(k) + q] = uu[q];
        }
    }
    for (int a = 0; a < 3; ++a) {
        box[6 * static_cast<size_t>(k) + a] = lo[a];
        box[6 * static_cast<size_t>(k) + 3 + a] = hi[a];
    }
    rec[3 * static_cast<size_t>(k)] = r0;
    rec[3 * static_cast<size_t>(k) + 1] = r1;
    rec[3 * static_cast<size_t>(k) + 2] = r2;
}

__global__ void k_permute(const float4* __restrict__ rec, const uint32_t* __restrict__ tn,
                          const uint32_t* __restrict__ tu, const uint32_t* __restrict__ perm, uint32_t n,
                          float4* __restrict__ rec_out, uint32_t* __restrict__ tn_out, uint32_t* __restrict__ tu_out) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t s = perm[k];
    for (int q = 0; q < 3; ++q) rec_out[3 * static_cast<size_t>(k) + q] = rec[3 * static_cast<size_t>(s) + q];
    if (tn)
        for (int q = 0; q < 3; ++q) tn_out[3 * static_cast<size_t>(k) + q] = tn[3 * static_cast<size_t>(s) + q];
    if (tu)
        for (int q = 0; q < 3; ++q) tu_out[3 * static_cast<size_t>(k) + q] = tu[3 * static_cast<size_t>(s) + q];
}

}  // namespace

}  // namespace gr

#include "sah_build.cuh"

namespace gr {

namespace {

// Device memory for the build alone, allocated and freed in the order of its stream, from a
// pool: cudaFree waits for all work on the device, so a creation would wait for every render
// that other threads have running.
struct StreamBuf {
    cudaStream_t st;
    void* ptr = nullptr;
    explicit StreamBuf(cudaStream_t s) : st(s) {}
    StreamBuf(const StreamBuf&) = delete;
    StreamBuf& operator=(const StreamBuf&) = delete;
    ~StreamBuf() { release(); }
    void release() {
        if (ptr) cudaFreeAsync(ptr, st);
        ptr = nullptr;
    }
    cudaError_t allocate(size_t bytes) {
        release();
        if (alloc_should_fail()) return cudaErrorMemoryAllocation;
        cudaMemPool_t pool;
        cudaError_t e = device_work().scratch.get(pool);
        if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&ptr, bytes, pool, st);
        if (e != cudaSuccess) ptr = nullptr;
        return e;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(ptr);
    }
};

// One allocation carved into the build's scratch buffers: sizes are added first, then
// reserve() makes the pointers valid.
struct Slab {
    StreamBuf buf;
    size_t total = 0;
    explicit Slab(cudaStream_t st) : buf(st) {}
    size_t add(size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) & ~size_t(255);
        return at;
    }
    cudaError_t reserve() { return buf.allocate(std::max<size_t>(total, 256)); }
    template <class T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(buf.as<unsigned char>() + offset);
    }
};

template <class T>
cudaError_t put(void* dst, const T* src, size_t count, cudaStream_t st) {
    if (!count) return cudaSuccess;
    return cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyHostToDevice, st);
}

// The order and the binary tree of the SAH build (sah_build.cuh): the host launches levels
// of large nodes, SAH_LEVELS_FIRST of them (15 for 102,400 triangles), then SAH_LEVELS_MORE at a time.
constexpr uint32_t SAH_LEVELS_FIRST = 16, SAH_LEVELS_MORE = 4;

struct SahScratch {
    size_t ctl, order[2], bucket, moved, tile_left, best, left, small;
    size_t nodes[2], tables[2], first_out[2], tile0[2], tiles[2];
    uint32_t max_big, max_tiles, max_small;
    SahScratch(Slab& m, uint32_t n) {
        max_big = n / (sah_small(n) + 1) + 1;
        max_tiles = n / SAH_TILE + max_big + 1;
        max_small = 2 * SAH_LEVELS * max_big;  // every large node leaves two at most
        ctl = m.add(sizeof(SahCtl));
        for (int k = 0; k < 2; ++k) {
            order[k] = m.add(n * sizeof(uint32_t));
            nodes[k] = m.add(max_big * sizeof(SahNode));
            tables[k] = m.add(size_t(max_big) * SAH_BUCKETS * SAH_VALUES * sizeof(int));
            first_out[k] = m.add(max_big * sizeof(uint32_t));
            tile0[k] = m.add(max_big * sizeof(uint32_t));
            tiles[k] = m.add(max_tiles * sizeof(uint2));
        }
        bucket = m.add(n);
        moved = m.add(n * sizeof(uint32_t));
        tile_left = m.add(max_tiles * sizeof(uint32_t));
        best = m.add(max_big * sizeof(uint32_t));
        left = m.add(max_big * sizeof(uint32_t));
        small = m.add(max_small * sizeof(SahSmall));
    }
    SahView view(const Slab& m, const float* box, Opened* opened, uint32_t n) const {
        SahView v;
        v.ctl = m.at<SahCtl>(ctl);
        v.box = box;
        for (int k = 0; k < 2; ++k) {
            v.order[k] = m.at<uint32_t>(order[k]);
            v.level[k] = SahLevel{m.at<SahNode>(nodes[k]), m.at<int>(tables[k]), m.at<uint32_t>(first_out[k]),
                                  m.at<uint32_t>(tile0[k]), m.at<uint2>(tiles[k])};
        }
        v.bucket = m.at<uint8_t>(bucket);
        v.moved = m.at<uint32_t>(moved);
        v.tile_left = m.at<uint32_t>(tile_left);
        v.best = m.at<uint32_t>(best);
        v.left = m.at<uint32_t>(left);
        v.small = m.at<SahSmall>(small);
        v.opened = reinterpret_cast<float*>(opened);
        v.n = n;
        v.most_small = sah_small(n);
        v.max_big = max_big;
        v.max_tiles = max_tiles;
        v.max_small = max_small;
        return v;
    }
};

// GR_ERR_INTERNAL: the host build has to make this tree.
gr_status sah_tree(const SahView& v, uint32_t* perm, cudaStream_t st, int& root) {
    SahCtl h{};
    for (int a = 0; a < 12; ++a) h.bounds[a] = a / 3 % 2 ? static_cast<int>(0x80000000u) : 0x7FFFFFFF;
    GR_CUDA_TRY(cudaMemcpyAsync(v.ctl, &h, sizeof(h), cudaMemcpyHostToDevice, st));
    const uint32_t sms = static_cast<uint32_t>(device_sm_count());
    k_sah_bounds<<<std::min((v.n + BB - 1) / BB, sms * 4u), BB, 0, st>>>(v);
    GR_CUDA_TRY(cudaGetLastError());
    k_sah_root<<<1, 32, 0, st>>>(v);
    GR_CUDA_TRY(cudaGetLastError());
    const uint32_t grid = std::min(v.max_tiles, sms * 8u);
    for (uint32_t level = 0;;) {
        const uint32_t stop = std::min(level + (level ? SAH_LEVELS_MORE : SAH_LEVELS_FIRST), SAH_LEVELS);
        for (; level < stop; ++level) {
            k_sah_buckets<<<grid, BB, 0, st>>>(v, level);
            k_sah_count<<<grid, BB, 0, st>>>(v, level);
            k_sah_front<<<grid, BB, 0, st>>>(v, level);
            k_sah_back<<<grid, BB, 0, st>>>(v, level);
            GR_CUDA_TRY(cudaGetLastError());
        }
        GR_CUDA_TRY(cudaMemcpyAsync(&h, v.ctl, sizeof(h), cudaMemcpyDeviceToHost, st));
        GR_CUDA_TRY(cudaStreamSynchronize(st));
        if (h.failed || (h.big[level] && level == SAH_LEVELS)) {
            set_error("device BVH build: left to the host");
            return GR_ERR_INTERNAL;
        }
        if (h.big[level] == 0) break;
    }
    if (v.most_small == SAH_SMALL_FEW)
        k_sah_small<SAH_SMALL_FEW>
            <<<std::min(h.small, sms * 8u), BB, sizeof(SahTree<SAH_SMALL_FEW>), st>>>(v, perm);
    else
        k_sah_small<SAH_SMALL_MANY>
            <<<std::min(h.small, sms * 4u), BB, sizeof(SahTree<SAH_SMALL_MANY>), st>>>(v, perm);
    GR_CUDA_TRY(cudaGetLastError());
    root = h.root;
    return GR_OK;
}

// Levels launched before the host looks how many there were (18 for 400,000 triangles; an
// empty level costs its launch).  A read-back per level and one launch per level for the
// stack use took 930 us there, this way 330.
constexpr uint32_t LEVELS_AT_ONCE = 22;

// `root_ref`: the binary tree's root node (of a single component: its leaf, ~0).  `nodes` has
// room for n: every wide node stands for a distinct binary node (or the root leaf).
template <int W>
gr_status collapse_levels(int root_ref, uint32_t n, CollapseCtl* ctl, const int* err, int4* todo, const Opened* opened,
                          const float* box, const uint32_t* perm, uint32_t leaf_size, float* nodes,
                          cudaStream_t st, uint32_t& num_wide, uint32_t& stack_depth) {
    const int4 root = make_int4(root_ref, 0, static_cast<int>(n), 0);
    const uint32_t one = 1;
    GR_CUDA_TRY(cudaMemsetAsync(ctl, 0, sizeof(CollapseCtl), st));
    GR_CUDA_TRY(cudaMemcpyAsync(ctl->count, &one, sizeof(one), cudaMemcpyHostToDevice, st));
    GR_CUDA_TRY(cudaMemcpyAsync(todo, &root, sizeof(root), cudaMemcpyHostToDevice, st));
    const uint32_t most = std::min((n + BB - 1) / BB, static_cast<uint32_t>(device_sm_count()) * 4u);
    CollapseCtl h;
    uint64_t width = 1;  // nodes a level can have
    for (uint32_t level = 0; level < MAX_LEVELS;) {
        const uint32_t stop = std::min(level + LEVELS_AT_ONCE, MAX_LEVELS);
        for (; level < stop; ++level) {
            const uint32_t grid = std::min<uint64_t>(most, (width + BB - 1) / BB);
            k_collapse<W><<<grid, BB, 0, st>>>(ctl, err, level, todo, opened, box, perm, leaf_size, nodes, n);
            GR_CUDA_TRY(cudaGetLastError());
            width = std::min<uint64_t>(width * W, n);
        }
        GR_CUDA_TRY(cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st));
        GR_CUDA_TRY(cudaStreamSynchronize(st));
        if (h.count[level] == 0) break;
    }
    if (h.count[MAX_LEVELS] != 0) {
        set_error("device BVH build: collapse did not terminate");
        return GR_ERR_INTERNAL;
    }
    num_wide = 0;
    for (uint32_t l = 0; l < MAX_LEVELS; ++l) num_wide += h.count[l];
    stack_depth = h.stack + 1;
    return GR_OK;
}

}  // namespace

gr_status build_bvh_device(const gr_scene_desc& desc, const HostBuild& h, SceneBuffers& b, cudaStream_t st,
                           uint32_t& num_wide, uint32_t& stack_depth, uint64_t& num_binary, uint64_t& bytes) {
    const uint32_t n = static_cast<uint32_t>(h.num_components);
    const uint32_t W = h.width, L = h.leaf_size;
    const uint32_t ni = n > 1 ? n - 1 : 1;  // internal nodes
    const uint32_t blocks = (n + BB - 1) / BB;
    size_t tmp_bytes = 0;
    if (!h.device_sah)
        GR_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, static_cast<uint32_t*>(nullptr),
                                                static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                                static_cast<uint32_t*>(nullptr), static_cast<int>(n), 0, 30, st));
    Slab m(st);
    const size_t o_box = m.add(size_t(n) * 6 * sizeof(float)), o_rec = m.add(size_t(n) * 3 * sizeof(float4));
    const size_t attr = size_t(n) * 3 * sizeof(uint32_t);
    const size_t o_tn = m.add(h.any_normals ? attr : 0), o_tu = m.add(h.any_uvs ? attr : 0);
    const size_t o_err = m.add(sizeof(int)), o_perm = m.add(n * sizeof(uint32_t));
    const size_t o_opened = m.add(size_t(ni) * sizeof(Opened));
    const size_t o_ctl = m.add(sizeof(CollapseCtl)), o_todo = m.add(size_t(n) * sizeof(int4));
    // Of the linear build, or of the SAH build.
    const size_t lin = h.device_sah ? 0 : n, lin_i = h.device_sah ? 0 : ni;
    const size_t o_bounds = m.add(6 * sizeof(int));
    const size_t o_code = m.add(lin * sizeof(uint32_t)), o_index = m.add(lin * sizeof(uint32_t));
    const size_t o_code_s = m.add(lin * sizeof(uint32_t)), o_tmp = m.add(std::max<size_t>(tmp_bytes, 16));
    const size_t o_split = m.add(lin_i * sizeof(int4)), o_par_i = m.add(lin_i * sizeof(int));
    const size_t o_par_l = m.add(lin * sizeof(int)), o_visits = m.add(lin_i * sizeof(int));
    // The SAH scene keeps as many nodes as there are; the linear one the worst case's room.
    const size_t node_bytes = size_t(8) * W * sizeof(float);
    const size_t o_nodes = m.add(h.device_sah ? n * node_bytes : 0);
    std::unique_ptr<SahScratch> sah;
    if (h.device_sah) sah.reset(new SahScratch(m, n));
    // The caller's arrays (records made on the device).
    std::vector<PrimSrc> src;
    std::vector<size_t> o_arrays;
    size_t o_src = 0;
    if (h.device_records) {
        o_src = m.add(desc.num_prims * sizeof(PrimSrc));
        for (uint32_t p = 0; p < desc.num_prims; ++p) {
            const gr_prim_desc& d = desc.prims[p];
            const bool mesh = d.kind == GR_PRIM_MESH;
            o_arrays.push_back(m.add(mesh ? size_t(d.num_vertices) * 3 * sizeof(float) : 0));
            o_arrays.push_back(m.add(mesh ? size_t(d.num_tris) * 3 * sizeof(uint32_t) : 0));
            o_arrays.push_back(m.add(mesh && d.tri_normals ? size_t(d.num_tris) * 3 * sizeof(uint32_t) : 0));
            o_arrays.push_back(m.add(mesh && d.tri_uvs ? size_t(d.num_tris) * 3 * sizeof(uint32_t) : 0));
        }
    }
    GR_CUDA_TRY(m.reserve());
    float* box = m.at<float>(o_box);
    float4* rec = m.at<float4>(o_rec);
    uint32_t* tn = h.any_normals ? m.at<uint32_t>(o_tn) : nullptr;
    uint32_t* tu = h.any_uvs ? m.at<uint32_t>(o_tu) : nullptr;
    int* err = m.at<int>(o_err);
    uint32_t* perm = m.at<uint32_t>(o_perm);
    GR_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
    if (h.device_records) {
        uint32_t first = 0;
        for (uint32_t p = 0; p < desc.num_prims; ++p) {
            const gr_prim_desc& d = desc.prims[p];
            PrimSrc q{};
            q.first = first;
            if (d.kind == GR_PRIM_SPHERE) {
                q.sphere = 1;
                for (int a = 0; a < 3; ++a) q.center[a] = d.center[a];
                q.radius = d.radius;
                first += 1;
            } else {
                const size_t* o = &o_arrays[4 * p];
                const size_t idx = size_t(d.num_tris) * 3;
                GR_CUDA_TRY(put(m.at<float>(o[0]), d.vertices, size_t(d.num_vertices) * 3, st));
                GR_CUDA_TRY(put(m.at<uint32_t>(o[1]), d.tri_vertices, idx, st));
                q.vertices = m.at<float>(o[0]);
                q.tris = m.at<uint32_t>(o[1]);
                q.num_vertices = d.num_vertices;
                if (d.tri_normals) {
                    GR_CUDA_TRY(put(m.at<uint32_t>(o[2]), d.tri_normals, idx, st));
                    q.tri_normals = m.at<uint32_t>(o[2]);
                    q.num_normals = d.num_normals;
                    q.nbase = h.nbase[p];
                }
                if (d.tri_uvs) {
                    GR_CUDA_TRY(put(m.at<uint32_t>(o[3]), d.tri_uvs, idx, st));
                    q.tri_uvs = m.at<uint32_t>(o[3]);
                    q.num_uvs = d.num_uvs;
                    q.ubase = h.ubase[p];
                }
                first += d.num_tris;
            }
            src.push_back(q);
        }
        GR_CUDA_TRY(put(m.at<PrimSrc>(o_src), src.data(), src.size(), st));
        k_records<<<blocks, BB, 0, st>>>(m.at<PrimSrc>(o_src), desc.num_prims, n, box, rec, tn, tu, err);
        GR_CUDA_TRY(cudaGetLastError());
    } else {
        GR_CUDA_TRY(put(box, h.item_boxes.data(), h.item_boxes.size(), st));
        GR_CUDA_TRY(put(reinterpret_cast<float*>(rec), h.prims.data(), h.prims.size(), st));
        GR_CUDA_TRY(put(tn, h.tri_normal_idx.data(), h.tri_normal_idx.size(), st));
        GR_CUDA_TRY(put(tu, h.tri_uv_idx.data(), h.tri_uv_idx.size(), st));
    }
    Opened* opened = m.at<Opened>(o_opened);
    int root = n > 1 ? 0 : ~0;
    if (sah) {
        const gr_status built = sah_tree(sah->view(m, box, opened, n), perm, st, root);
        if (built != GR_OK) return built;
    } else {
        int init[6];
        for (int a = 0; a < 3; ++a) {
            init[a] = 0x7FFFFFFF;  // ordered(+max)
            init[3 + a] = static_cast<int>(0x80000000u);
        }
        int* bounds = m.at<int>(o_bounds);
        GR_CUDA_TRY(cudaMemcpyAsync(bounds, init, sizeof(init), cudaMemcpyHostToDevice, st));
        const uint32_t grid = std::min(blocks, static_cast<uint32_t>(device_sm_count()) * 4u);
        k_centroid_bounds<<<grid, BB, 0, st>>>(box, n, bounds);
        GR_CUDA_TRY(cudaGetLastError());
        uint32_t *code = m.at<uint32_t>(o_code), *index = m.at<uint32_t>(o_index), *code_s = m.at<uint32_t>(o_code_s);
        k_morton<<<blocks, BB, 0, st>>>(box, n, bounds, code, index);
        GR_CUDA_TRY(cudaGetLastError());
        GR_CUDA_TRY(cub::DeviceRadixSort::SortPairs(m.at<void>(o_tmp), tmp_bytes, code, code_s, index, perm,
                                                    static_cast<int>(n), 0, 30, st));
        int *par_i = m.at<int>(o_par_i), *par_l = m.at<int>(o_par_l), *visits = m.at<int>(o_visits);
        int4* split = m.at<int4>(o_split);
        GR_CUDA_TRY(cudaMemsetAsync(par_i, 0xFF, ni * sizeof(int), st));  // root: -1
        GR_CUDA_TRY(cudaMemsetAsync(par_l, 0xFF, n * sizeof(int), st));
        GR_CUDA_TRY(cudaMemsetAsync(visits, 0, ni * sizeof(int), st));
        if (n > 1) {
            k_radix_tree<<<(n - 1 + BB - 1) / BB, BB, 0, st>>>(code_s, static_cast<int>(n), split, par_i, par_l);
            GR_CUDA_TRY(cudaGetLastError());
            k_boxes<<<blocks, BB, 0, st>>>(box, perm, static_cast<int>(n), split, par_i, par_l, opened, visits, err);
            GR_CUDA_TRY(cudaGetLastError());
        }
    }
    int e = 0;
    GR_CUDA_TRY(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    CollapseCtl* ctl = m.at<CollapseCtl>(o_ctl);
    int4* todo = m.at<int4>(o_todo);
    if (!sah) GR_CUDA_TRY(b.nodes.ensure(n * node_bytes));
    float* nodes = sah ? m.at<float>(o_nodes) : b.nodes.as<float>();
    auto collapse = W == 2 ? collapse_levels<2> : (W == 8 ? collapse_levels<8> : collapse_levels<4>);
    const gr_status s = collapse(root, n, ctl, err, todo, opened, box, perm, L, nodes, st, num_wide, stack_depth);
    if (s != GR_OK) return s;  // (it has synchronised the stream, so `e` is there)
    if (e == ERR_BAD_INDEX) {
        set_error("device BVH build: an index is out of range");
        return GR_ERR_INVALID_ARGUMENT;
    }
    if (e) {
        set_error("device BVH build: inconsistent radix tree");
        return GR_ERR_INTERNAL;
    }
    if (stack_depth > static_cast<uint32_t>(MAX_STACK)) {
        set_error("device BVH build: the tree needs a traversal stack of " + std::to_string(stack_depth) +
                  " entries (limit " + std::to_string(MAX_STACK) + ")");
        return GR_ERR_STACK_OVERFLOW;
    }
    if (sah) {
        SahCtl ctl_end;
        GR_CUDA_TRY(b.nodes.ensure(num_wide * node_bytes));
        GR_CUDA_TRY(cudaMemcpyAsync(b.nodes.ptr, nodes, num_wide * node_bytes, cudaMemcpyDeviceToDevice, st));
        GR_CUDA_TRY(cudaMemcpyAsync(&ctl_end, m.at<SahCtl>(sah->ctl), sizeof(ctl_end), cudaMemcpyDeviceToHost, st));
        GR_CUDA_TRY(cudaStreamSynchronize(st));
        if (ctl_end.failed) {
            set_error("device BVH build: left to the host");
            return GR_ERR_INTERNAL;
        }
        num_binary = 2 * (uint64_t(n) - ctl_end.excess) - 1;
    }
    const size_t rec_bytes = size_t(n) * 3 * sizeof(float4);
    GR_CUDA_TRY(b.prims.ensure(rec_bytes));
    if (tn) GR_CUDA_TRY(b.tri_nidx.ensure(attr));
    if (tu) GR_CUDA_TRY(b.tri_uvidx.ensure(attr));
    k_permute<<<blocks, BB, 0, st>>>(rec, tn, tu, perm, n, b.prims.as<float4>(), b.tri_nidx.as<uint32_t>(),
                                     b.tri_uvidx.as<uint32_t>());
    GR_CUDA_TRY(cudaGetLastError());
    m.buf.release();  // (goes back to the device with the wait)
    GR_CUDA_TRY(cudaStreamSynchronize(st));
    bytes += num_wide * node_bytes + rec_bytes + (tn ? attr : 0) + (tu ? attr : 0);
    return GR_OK;
}

gr_status build_index_check() {
#if GR_CHECKED
    bool bad = false;
    GR_CUDA_TRY(take_bad_index(bad));
    if (bad) {
        set_error("device BVH build: an index was out of range (checked build)");
        return GR_ERR_INTERNAL;
    }
#endif
    return GR_OK;
}

}  // namespace gr
