// CWBVH built on the GPU from device-resident triangles, for scenes that must
// be ready quickly (a new scene admitted into a server) rather than traced
// at the best speed: a binary BVH over the Morton-ordered triangles (Karras's
// radix tree, or locally-ordered clustering), optional treelet passes, then
// a cost-optimal collapse into 8-wide nodes written directly in the CWBVH
// node format, with Woop rows and the primitive map, all on one stream.
//
//  1. centroid bounds (reduction), Morton code of each centroid above the
//     triangle number (unique 64-bit keys: ceil(log2 n) index bits, the rest,
//     up to 21 per axis, for the code), radix sort;
//  2. the binary tree: either internal node i of the radix tree over the
//     sorted keys, its key range and split from the longest common prefixes
//     (Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees,
//     and k-d Trees", HPG 2012), with boxes and triangle counts bottom-up
//     (each leaf walks to the root and the second thread to reach a node
//     completes it, one atomic per node); or rounds of locally-ordered
//     clustering (see ploc_tree);
//  3. optional treelet restructuring passes (see restructure);
//  4. the host builder's cost-optimal collapse (dynamic programme over 1..8
//     slots per binary node, bottom-up), then level by level from the root
//     each 8-wide node's slots as it chose them; children with at most 3
//     triangles become leaves, the others 8-wide nodes of the next level.
//     Slots are assigned by the same octant rule as the host converter,
//     boxes quantized the same way, inner children get one contiguous block
//     and leaf triangles one contiguous run per node.
//
// The tree is a valid CWBVH for every trace kernel; it is not the host
// builder's (no spatial splits, different binary tree), so traversal is
// slower and the bytes differ.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "runtime.h"

namespace rq {
namespace {

// A box with the SAH cost and the triangle count of what it bounds: two
// 16-byte loads give all that a walk up the tree reads of a child.
struct __align__(16) NodeBox {
    float lo[3];
    float cost;  // SAH cost of the subtree
    float hi[3];
    int32_t count;  // triangles below
};

struct __align__(16) BNode {
    int32_t left, right;  // >= 0: internal node, < 0: leaf ~(sorted position)
    int32_t parent;       // -1 at the root
    uint32_t stamps;      // treelet passes (from 1): low half the last that rewrote this node, high half the
                          // last that rewrote this node or one below it on its way up
    NodeBox b;
};
static_assert(sizeof(NodeBox) == 32 && sizeof(BNode) == 48, "node layout");

// SAH weights of the treelet restructuring (Karras and Aila 2013).
constexpr float kCt = 1.2f;  // per node
constexpr float kCi = 1.0f;  // per triangle

__device__ inline unsigned f2ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ inline float ord2f(unsigned u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u); }

__device__ inline float3 vtx(const float* v, int32_t k) {
    const int64_t o = 3 * (int64_t)k;
    return make_float3(v[o], v[o + 1], v[o + 2]);
}

__device__ inline void tri_box(const float* v, const int32_t* idx, int64_t t, float lo[3], float hi[3]) {
    const float3 a = vtx(v, idx[3 * t]), b = vtx(v, idx[3 * t + 1]), c = vtx(v, idx[3 * t + 2]);
    lo[0] = fminf(a.x, fminf(b.x, c.x)); hi[0] = fmaxf(a.x, fmaxf(b.x, c.x));
    lo[1] = fminf(a.y, fminf(b.y, c.y)); hi[1] = fmaxf(a.y, fmaxf(b.y, c.y));
    lo[2] = fminf(a.z, fminf(b.z, c.z)); hi[2] = fmaxf(a.z, fmaxf(b.z, c.z));
}

// Sets *bad when an index is outside [0, nv): nothing else reads vertices
// through indices that have not passed this check.
__global__ void check_indices_kernel(const int32_t* idx, int64_t n3, int64_t nv, unsigned* bad) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n3; q += (int64_t)gridDim.x * blockDim.x)
        if (idx[q] < 0 || (int64_t)idx[q] >= nv) atomicOr(bad, 1u);
}

// ---- Triangle pre-splitting (the splitting stage of Karras and Aila, "Fast
// Parallel Construction of High-Quality Bounding Volume Hierarchies", HPG
// 2013, section 5).  A triangle whose box is much larger than the triangle
// itself (a sliver lying across the axes) is cut into several references
// along the planes of a 1024^3 grid over the scene, the most important plane
// first, so that the tree stages see tight boxes.  Each triangle receives
// pieces in proportion to its priority (2^m * wasted area)^(1/3), where m is
// the Morton level of the most important grid plane its box crosses and the
// wasted area is its box's half area minus the least half area boxes of its
// pieces can reach; the budget caps the extra pieces.  The references go to
// the tree stages as a "box mesh": a reference with box [lo, hi] is the
// triangle (lo, hi, hi), whose bounds are that box, so those stages read
// reference boxes through the same code as triangle boxes.  Only the Woop
// rows and the primitive map go back to the triangle.
constexpr int kSplitGridBits = 10;
constexpr int kMaxPieces = 32;

struct SplitGrid {
    float b0[3], ext[3];
};

__device__ inline SplitGrid split_grid(const unsigned* sb) {
    SplitGrid g;
    for (int a = 0; a < 3; ++a) {
        g.b0[a] = ord2f(sb[a]);
        g.ext[a] = ord2f(sb[3 + a]) - g.b0[a];
    }
    return g;
}

__device__ inline int grid_cell(const SplitGrid& g, int a, float x) {
    const float f = (x - g.b0[a]) / g.ext[a] * (float)(1 << kSplitGridBits);
    return (int)fminf(fmaxf(floorf(f), 0.f), (float)((1 << kSplitGridBits) - 1));
}

// The most important grid plane strictly inside [lo, hi]: the highest bit in
// which the cells of lo and hi differ, x before y before z at equal bits (the
// Morton order).  Returns its Morton level (3 * bit + 2 - axis) or -1.
__device__ int split_plane(const SplitGrid& g, const float lo[3], const float hi[3], int& axis, float& pos) {
    int best = -1;
    for (int a = 0; a < 3; ++a) {
        if (!(g.ext[a] > 0.f)) continue;
        const int q0 = grid_cell(g, a, lo[a]), q1 = grid_cell(g, a, hi[a]);
        if (q0 >= q1) continue;
        const int bit = 31 - __clz(q0 ^ q1);
        const int level = 3 * bit + 2 - a;
        if (level <= best) continue;
        const int cell = (q1 >> bit) << bit;  // first cell above the plane
        const float p = g.b0[a] + g.ext[a] * ((float)cell / (float)(1 << kSplitGridBits));
        if (!(p > lo[a] && p < hi[a])) continue;
        best = level;
        axis = a;
        pos = p;
    }
    return best;
}

// Scene bounds of the triangle boxes as order-preserving unsigned min / max.
__global__ void scene_bounds_kernel(const float* v, const int32_t* idx, int64_t n, unsigned* sb) {
    unsigned mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int32_t* ti = idx + 3 * t;
        for (int c = 0; c < 3; ++c) {
            const float3 p = vtx(v, ti[c]);
            const unsigned u[3] = {f2ord(p.x), f2ord(p.y), f2ord(p.z)};
            for (int a = 0; a < 3; ++a) {
                mn[a] = min(mn[a], u[a]);
                mx[a] = max(mx[a], u[a]);
            }
        }
    }
    for (int a = 0; a < 3; ++a)
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], o));
            mx[a] = max(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int a = 0; a < 3; ++a) {
            atomicMin(sb + a, mn[a]);
            atomicMax(sb + 3 + a, mx[a]);
        }
}

__device__ inline float half_area3(const float lo[3], const float hi[3]) {
    const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// Priority of each triangle.  The box of a piece of a flat patch with unit
// normal n and area A has half area at least 2 A (|nx| + |ny| + |nz|), which
// is |c.x| + |c.y| + |c.z| for the whole triangle, c = (b - a) x (c - a);
// the box's half area above that is what splitting can remove.
__global__ void split_priority_kernel(const float* v, const int32_t* idx, int64_t n, const unsigned* sb,
                                      float* prio) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int32_t* ti = idx + 3 * t;
    const float3 a = vtx(v, ti[0]), b = vtx(v, ti[1]), c = vtx(v, ti[2]);
    const float lo[3] = {fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z))};
    const float hi[3] = {fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z))};
    const float ex = b.x - a.x, ey = b.y - a.y, ez = b.z - a.z;
    const float fx = c.x - a.x, fy = c.y - a.y, fz = c.z - a.z;
    const float ideal = fabsf(ey * fz - ez * fy) + fabsf(ez * fx - ex * fz) + fabsf(ex * fy - ey * fx);
    const float waste = half_area3(lo, hi) - ideal;
    const SplitGrid g = split_grid(sb);
    int axis = 0;
    float pos = 0.f;
    const int level = split_plane(g, lo, hi, axis, pos);
    prio[t] = (level < 0 || !(waste > 0.f)) ? 0.f : exp2f((float)level / 3.f) * cbrtf(waste);
}

// Pieces per triangle: 1 + its share of the `extra` budget, at most kMaxPieces.
__global__ void split_count_kernel(const float* prio, int64_t n, const float* sum, double extra, int64_t* pieces) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double s = (double)*sum;
    const double share = s > 0.0 ? floor(extra * (double)prio[t] / s) : 0.0;
    pieces[t] = 1 + (int64_t)fmin(share, (double)(kMaxPieces - 1));
}

// The part of triangle (a, b, c) on one side of the plane x[axis] = p (upper
// side when `upper`), bounded in double and rounded outwards, clipped to box
// [blo, bhi].  Returns false when that part misses the box.
__device__ bool clip_side(const double3 (&tri)[3], int axis, double p, bool upper, const float blo[3],
                          const float bhi[3], float lo[3], float hi[3]) {
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    auto comp = [](const double3& q, int a) { return a == 0 ? q.x : (a == 1 ? q.y : q.z); };
    auto add = [&](double x, double y, double z) {
        mn[0] = fmin(mn[0], x); mx[0] = fmax(mx[0], x);
        mn[1] = fmin(mn[1], y); mx[1] = fmax(mx[1], y);
        mn[2] = fmin(mn[2], z); mx[2] = fmax(mx[2], z);
    };
    bool any = false;
    for (int i = 0; i < 3; ++i) {
        const double3& q = tri[i];
        const double qi = comp(q, axis);
        if (upper ? qi >= p : qi <= p) {
            add(q.x, q.y, q.z);
            any = true;
        }
        const double3& r = tri[(i + 1) % 3];
        const double ri = comp(r, axis);
        if ((qi < p && ri > p) || (qi > p && ri < p)) {
            const double s = (p - qi) / (ri - qi);
            double x = q.x + s * (r.x - q.x), y = q.y + s * (r.y - q.y), z = q.z + s * (r.z - q.z);
            if (axis == 0) x = p; else if (axis == 1) y = p; else z = p;
            add(x, y, z);
            any = true;
        }
    }
    if (!any) return false;
    for (int a = 0; a < 3; ++a) {
        lo[a] = fmaxf(__double2float_rd(mn[a]), blo[a]);
        hi[a] = fminf(__double2float_ru(mx[a]), bhi[a]);
        if (!(lo[a] <= hi[a])) return false;
    }
    return true;
}

// Cuts triangle t into pieces[t] references at off[t]: the box mesh (two
// corners per reference in rv, the triangle (2r, 2r + 1, 2r + 1) in ri) and
// the triangle of each reference (rtri).  Pieces are taken depth-first, the
// plane of each cut by split_plane, the pieces of a box shared between its
// two sides by their half areas; a box no plane cuts is one reference and
// any slots left over repeat the last reference.
struct SplitEntry {
    float lo[3], hi[3];
    int count;
};

__global__ void split_kernel(const float* v, const int32_t* idx, int64_t n, const unsigned* sb,
                             const int64_t* pieces, const int64_t* off, float* rv, int32_t* ri, int32_t* rtri) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int32_t* ti = idx + 3 * t;
    double3 tri[3];
    float lo[3], hi[3];
    for (int c = 0; c < 3; ++c) {
        const float3 p = vtx(v, ti[c]);
        tri[c] = make_double3(p.x, p.y, p.z);
    }
    for (int a = 0; a < 3; ++a) {
        const float x0 = a == 0 ? (float)tri[0].x : (a == 1 ? (float)tri[0].y : (float)tri[0].z);
        const float x1 = a == 0 ? (float)tri[1].x : (a == 1 ? (float)tri[1].y : (float)tri[1].z);
        const float x2 = a == 0 ? (float)tri[2].x : (a == 1 ? (float)tri[2].y : (float)tri[2].z);
        lo[a] = fminf(x0, fminf(x1, x2));
        hi[a] = fmaxf(x0, fmaxf(x1, x2));
    }
    const int total = (int)(pieces[t] < kMaxPieces ? pieces[t] : kMaxPieces);
    const int64_t base = off[t];
    const SplitGrid g = split_grid(sb);
    SplitEntry st[kMaxPieces];
    int sp = 0, emitted = 0, steps = 0;
    st[sp++] = SplitEntry{{lo[0], lo[1], lo[2]}, {hi[0], hi[1], hi[2]}, total};
    float last[6] = {lo[0], lo[1], lo[2], hi[0], hi[1], hi[2]};
    auto emit = [&](const float* elo, const float* ehi) {
        if (emitted >= total) return;
        const int64_t r = base + emitted++;
        for (int a = 0; a < 3; ++a) {
            rv[6 * r + a] = elo[a];
            rv[6 * r + 3 + a] = ehi[a];
            last[a] = elo[a];
            last[3 + a] = ehi[a];
        }
        ri[3 * r] = (int32_t)(2 * r);
        ri[3 * r + 1] = (int32_t)(2 * r + 1);
        ri[3 * r + 2] = (int32_t)(2 * r + 1);
        rtri[r] = (int32_t)t;
    };
    while (sp > 0 && emitted < total) {
        const SplitEntry e = st[--sp];
        int axis = 0;
        float pos = 0.f;
        if (e.count == 1 || ++steps > 4 * kMaxPieces || split_plane(g, e.lo, e.hi, axis, pos) < 0) {
            emit(e.lo, e.hi);
            continue;
        }
        SplitEntry L, R;
        const bool okl = clip_side(tri, axis, (double)pos, false, e.lo, e.hi, L.lo, L.hi);
        const bool okr = clip_side(tri, axis, (double)pos, true, e.lo, e.hi, R.lo, R.hi);
        if (!okl && !okr) {
            emit(e.lo, e.hi);
            continue;
        }
        if (!okl || !okr) {  // all pieces to the one side that holds the triangle
            SplitEntry& o = okl ? L : R;
            o.count = e.count;
            st[sp++] = o;
            continue;
        }
        const float al = half_area3(L.lo, L.hi), ar = half_area3(R.lo, R.hi);
        int cl = (al + ar > 0.f) ? __float2int_rn((float)e.count * al / (al + ar)) : e.count / 2;
        cl = max(1, min(e.count - 1, cl));
        L.count = cl;
        R.count = e.count - cl;
        st[sp++] = R;  // counts on the stack never exceed total <= kMaxPieces entries
        st[sp++] = L;
    }
    while (emitted < total) emit(last, last + 3);
}

// Centroid bounds as order-preserving unsigned min / max (6 words).
__global__ void centroid_bounds_kernel(const float* v, const int32_t* idx, int64_t n, unsigned* ob) {
    unsigned mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        float lo[3], hi[3];
        tri_box(v, idx, t, lo, hi);
        for (int a = 0; a < 3; ++a) {
            const unsigned c = f2ord(0.5f * (lo[a] + hi[a]));
            mn[a] = min(mn[a], c);
            mx[a] = max(mx[a], c);
        }
    }
    for (int a = 0; a < 3; ++a)
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xFFFFFFFFu, mn[a], o));
            mx[a] = max(mx[a], __shfl_xor_sync(0xFFFFFFFFu, mx[a], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int a = 0; a < 3; ++a) {
            atomicMin(ob + a, mn[a]);
            atomicMax(ob + 3 + a, mx[a]);
        }
}

// Spreads the low 21 bits of x to every third bit.
__device__ inline uint64_t spread3(uint64_t x) {
    x &= 0x1FFFFFull;
    x = (x | (x << 32)) & 0x001F00000000FFFFull;
    x = (x | (x << 16)) & 0x001F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// key = Morton code of the centroid (`axis_bits` per axis) above the
// triangle number (`idx_bits`): unique, and as fine a grid as 64 bits allow.
__global__ void morton_kernel(const float* v, const int32_t* idx, int64_t n, const unsigned* ob, int axis_bits,
                              int idx_bits, uint64_t* keys) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    float lo[3], hi[3];
    tri_box(v, idx, t, lo, hi);
    const float cells = (float)(1u << axis_bits);
    uint64_t q[3];
    for (int a = 0; a < 3; ++a) {
        const float b0 = ord2f(ob[a]), b1 = ord2f(ob[3 + a]);
        const float ext = b1 - b0;
        float f = ext > 0.f ? (0.5f * (lo[a] + hi[a]) - b0) / ext : 0.f;
        f = fminf(fmaxf(f, 0.f), 1.f);
        q[a] = min((uint64_t)((1u << axis_bits) - 1), (uint64_t)(f * cells));
    }
    const uint64_t m = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    keys[t] = (m << idx_bits) | (uint64_t)t;
}

__device__ inline int delta(const uint64_t* k, int64_t n, int64_t i, int64_t j) {
    if (j < 0 || j >= n) return -1;
    return __clzll((long long)(k[i] ^ k[j]));
}

// Internal node i of the radix tree (Karras 2012, section 4).
__global__ void radix_tree_kernel(const uint64_t* k, int64_t n, BNode* nodes, int32_t* leaf_parent) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = delta(k, n, i, i + 1) - delta(k, n, i, i - 1) >= 0 ? 1 : -1;
    const int dmin = delta(k, n, i, i - d);
    int64_t lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax *= 2;
    int64_t l = 0;
    for (int64_t t = lmax / 2; t >= 1; t /= 2)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int64_t j = i + l * d;
    const int dnode = delta(k, n, i, j);
    int64_t s = 0;
    for (int64_t div = 2;; div *= 2) {
        const int64_t t = (l + div - 1) / div;
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
    }
    const int64_t gamma = i + s * d + min(d, 0);
    const int64_t lo = min(i, j), hi = max(i, j);
    BNode& nd = nodes[i];
    nd.left = lo == gamma ? ~(int32_t)gamma : (int32_t)gamma;
    nd.right = hi == gamma + 1 ? ~(int32_t)(gamma + 1) : (int32_t)(gamma + 1);
    if (nd.left >= 0) nodes[nd.left].parent = (int32_t)i;
    else leaf_parent[gamma] = (int32_t)i;
    if (nd.right >= 0) nodes[nd.right].parent = (int32_t)i;
    else leaf_parent[gamma + 1] = (int32_t)i;
    if (i == 0) nd.parent = -1;
    nd.stamps = 0u;
}

// The triangle of a sorted key: its low idx_bits bits (idx_mask).
__device__ inline int64_t key_tri(const uint64_t* k, int64_t pos, uint64_t idx_mask) {
    return (int64_t)(k[pos] & idx_mask);
}

// Half the surface area of a box, and the SAH cost of a node over its two
// children, with every rounding explicit: the treelet kernels (one thread or
// one warp per treelet) compute the same costs bit for bit.
__device__ inline float half_area(const float lo[3], const float hi[3]) {
    const float dx = __fsub_rn(hi[0], lo[0]), dy = __fsub_rn(hi[1], lo[1]), dz = __fsub_rn(hi[2], lo[2]);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}
__device__ inline float node_cost(float area, float c0, float c1) {
    return __fadd_rn(__fadd_rn(__fmul_rn(kCt, area), c0), c1);
}

// The box of a child: a node's, or that of the leaf at a sorted position.
// Boxes other threads of the same launch may have written are read from L2
// (ld.cg), never from a possibly stale L1 line.
__device__ inline NodeBox child_box(const BNode* nodes, const NodeBox* leaves, int32_t code) {
    const float4* p = reinterpret_cast<const float4*>(code >= 0 ? &nodes[code].b : &leaves[~code]);
    const float4 x = __ldcg(p), y = __ldcg(p + 1);
    NodeBox b;
    b.lo[0] = x.x; b.lo[1] = x.y; b.lo[2] = x.z; b.cost = x.w;
    b.hi[0] = y.x; b.hi[1] = y.y; b.hi[2] = y.z; b.count = __float_as_int(y.w);
    return b;
}
__device__ inline void store_box(NodeBox* to, const NodeBox& b) {
    float4* p = reinterpret_cast<float4*>(to);
    p[0] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.cost);
    p[1] = make_float4(b.hi[0], b.hi[1], b.hi[2], __int_as_float(b.count));
}
// The box of a node over two children, its count and its cost.
__device__ inline NodeBox join(const NodeBox& l, const NodeBox& r) {
    NodeBox b;
    for (int a = 0; a < 3; ++a) {
        b.lo[a] = fminf(l.lo[a], r.lo[a]);
        b.hi[a] = fmaxf(l.hi[a], r.hi[a]);
    }
    b.count = l.count + r.count;
    b.cost = node_cost(half_area(b.lo, b.hi), l.cost, r.cost);
    return b;
}

// The boxes of the leaves in sorted order.
__global__ void leaf_boxes_kernel(const uint64_t* k, uint64_t idx_mask, int64_t n, const float* v, const int32_t* idx,
                                  NodeBox* leaves) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    NodeBox b;
    tri_box(v, idx, key_tri(k, p, idx_mask), b.lo, b.hi);
    b.cost = __fmul_rn(kCi, half_area(b.lo, b.hi));
    b.count = 1;
    store_box(leaves + p, b);
}

// Boxes and counts bottom-up: the second of a node's two children to arrive
// completes it and goes on to the parent.
__global__ void boxes_kernel(int64_t n, const NodeBox* leaves, BNode* nodes, const int32_t* leaf_parent,
                             int32_t* arrivals) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int32_t node = leaf_parent[p];
    while (node >= 0) {
        __threadfence();
        if (atomicAdd(&arrivals[node], 1) == 0) return;  // the sibling finishes this node
        __threadfence();
        store_box(&nodes[node].b, join(child_box(nodes, leaves, nodes[node].left),
                                       child_box(nodes, leaves, nodes[node].right)));
        node = nodes[node].parent;
    }
}

// ---- Treelet restructuring (Karras and Aila, "Fast Parallel Construction of
// High-Quality Bounding Volume Hierarchies", HPG 2013): bottom-up again, each
// node with at least `min_count` triangles forms a treelet by expanding its
// largest-area leaf until it has 7 leaves, finds the SAH-optimal binary tree
// over those leaves by dynamic programming over the 127 leaf subsets, and
// rebuilds the treelet with it (reusing its 6 internal nodes) when cheaper.
// Treelets of different nodes being restructured at once are disjoint: a node
// is processed only when both its children are final.
constexpr int kTreeletLeaves = 7;

// Links other threads of the same launch may have rewritten are read from L2.
__device__ inline int32_t ld_left(const BNode* nodes, int32_t x) { return __ldcg(&nodes[x].left); }
__device__ inline int32_t ld_right(const BNode* nodes, int32_t x) { return __ldcg(&nodes[x].right); }
__device__ inline int32_t ld_parent(const BNode* nodes, int32_t x) { return __ldcg(&nodes[x].parent); }

__device__ void restructure(BNode* nodes, const NodeBox* leaves, int32_t* leaf_parent, int32_t root) {
    int32_t inner[kTreeletLeaves - 1], leaf[kTreeletLeaves];
    float larea[kTreeletLeaves];
    int n_in = 1, n_leaf = 2;
    inner[0] = root;
    leaf[0] = ld_left(nodes, root);
    leaf[1] = ld_right(nodes, root);
    float llo[kTreeletLeaves][3], lhi[kTreeletLeaves][3], lcost[kTreeletLeaves];
    int32_t lcnt[kTreeletLeaves];
    auto take = [&](int q, int32_t code) {
        const NodeBox b = child_box(nodes, leaves, code);
        leaf[q] = code;
        for (int a = 0; a < 3; ++a) { llo[q][a] = b.lo[a]; lhi[q][a] = b.hi[a]; }
        lcost[q] = b.cost;
        lcnt[q] = b.count;
        larea[q] = half_area(b.lo, b.hi);
    };
    take(0, leaf[0]);
    take(1, leaf[1]);
    while (n_leaf < kTreeletLeaves) {
        int best = -1;
        float ba = -1.f;
        for (int q = 0; q < n_leaf; ++q)
            if (leaf[q] >= 0 && larea[q] > ba) { ba = larea[q]; best = q; }
        if (best < 0) break;
        const int32_t x = leaf[best];
        inner[n_in++] = x;
        const int32_t l = ld_left(nodes, x), r = ld_right(nodes, x);
        take(best, l);
        take(n_leaf, r);
        ++n_leaf;
    }
    if (n_leaf < 3) return;
    const int full = (1 << n_leaf) - 1;
    // Subset boxes are recomputed from the leaves when needed instead of
    // kept per subset: min / max are exact in any order, so the boxes are
    // the same, and the per-thread table shrinks from 3.7 KB to 640 B.
    auto subset_box = [&](int S, float lo[3], float hi[3]) {
        for (int a = 0; a < 3; ++a) { lo[a] = FLT_MAX; hi[a] = -FLT_MAX; }
        for (int q = 0; q < n_leaf; ++q)
            if (S & (1 << q))
                for (int a = 0; a < 3; ++a) { lo[a] = fminf(lo[a], llo[q][a]); hi[a] = fmaxf(hi[a], lhi[q][a]); }
    };
    float cost[1 << kTreeletLeaves];
    uint8_t part[1 << kTreeletLeaves];
    for (int S = 1; S <= full; ++S) {
        const int low = __ffs(S) - 1;
        const int rest = S & (S - 1);
        if (rest == 0) {
            cost[S] = lcost[low];
            part[S] = 0;
            continue;
        }
        float slo[3], shi[3];
        subset_box(S, slo, shi);
        float best = FLT_MAX;
        int bp = 0;
        // partitions {P, S \ P} with the lowest leaf in P, P != S
        for (int P = (S - 1) & S; P > 0; P = (P - 1) & S) {
            if (!(P & (1 << low))) continue;
            const float c = __fadd_rn(cost[P], cost[S ^ P]);
            if (c < best) { best = c; bp = P; }
        }
        cost[S] = __fadd_rn(__fmul_rn(kCt, half_area(slo, shi)), best);
        part[S] = (uint8_t)bp;
    }
    if (!(cost[full] < 0.999f * __ldcg(&nodes[root].b.cost))) return;
    // every subset the new tree splits must have a split (finite costs); check
    // before writing anything
    {
        int st[kTreeletLeaves], sp = 0;
        st[sp++] = full;
        while (sp > 0) {
            const int S = st[--sp];
            const int P = part[S];
            if (P == 0 || (P & ~S) != 0 || P == S) return;
            if (P & (P - 1)) st[sp++] = P;
            if ((S ^ P) & ((S ^ P) - 1)) st[sp++] = S ^ P;
            if (sp > kTreeletLeaves - 1) return;
        }
    }
    // rebuild top-down: subset -> node, internal nodes taken from `inner`
    int32_t st_set[kTreeletLeaves], st_node[kTreeletLeaves];
    int sp = 0, used = 1;
    st_set[sp] = full;
    st_node[sp++] = root;
    while (sp > 0) {
        --sp;
        const int S = st_set[sp];
        const int32_t nd = st_node[sp];
        const int P = part[S];
        const int side[2] = {P, S ^ P};
        int32_t code[2];
        for (int c = 0; c < 2; ++c) {
            const int T = side[c];
            if ((T & (T - 1)) == 0) {  // one leaf of the treelet
                code[c] = leaf[__ffs(T) - 1];
                if (code[c] >= 0) nodes[code[c]].parent = nd;
                else leaf_parent[~code[c]] = nd;
            } else {
                const int32_t ni = inner[used++];
                code[c] = ni;
                nodes[ni].parent = nd;
                st_set[sp] = T;
                st_node[sp++] = ni;
            }
        }
        BNode& b = nodes[nd];
        b.left = code[0];
        b.right = code[1];
        NodeBox nb;
        subset_box(S, nb.lo, nb.hi);
        nb.count = 0;
        for (int q = 0; q < n_leaf; ++q)
            if (S & (1 << q)) nb.count += lcnt[q];
        nb.cost = cost[S];
        store_box(&b.b, nb);
    }
}

__global__ void treelet_kernel(int64_t n, const NodeBox* leaves, BNode* nodes, int32_t* leaf_parent, int32_t* arrivals,
                               int min_count) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int32_t node = leaf_parent[p];
    while (node >= 0) {
        __threadfence();
        if (atomicAdd(&arrivals[node], 1) == 0) return;
        __threadfence();
        // this node's cost from its (final) children, then its treelet
        const NodeBox b = join(child_box(nodes, leaves, ld_left(nodes, node)),
                               child_box(nodes, leaves, ld_right(nodes, node)));
        __stcg(&nodes[node].b.cost, b.cost);
        if (b.count >= min_count) restructure(nodes, leaves, leaf_parent, node);
        node = ld_parent(nodes, node);
    }
}

// ---- The same restructuring with a warp per treelet (the parallel form of
// Karras and Aila, section 4.2).  Lanes walk up the tree as in
// treelet_kernel; at each step the nodes whose treelets are due are taken one
// at a time by the whole warp: lane q holds leaf q (its box and, ahead of its
// being opened, its links) while the treelet grows; the subsets of one size
// are costed by different lanes, smaller subsets first, so every partition's
// two parts are ready; the 31 partitions of a 6-leaf set are spread over four
// lanes and the 63 of the 7-leaf set over the warp; and a lane writes each
// node of the new treelet.  Every subset's cost is the same expression as in
// restructure(), over the same partitions (a subset's lowest leaf stays in P,
// the others run down through the subsets of the rest), and the chosen
// partition is the first minimum in its order there, so the trees are
// identical.
//
// From the second pass on a treelet is due only if its subtree is not the one
// that the pass before left its root with: that pass rewrote the root (by its
// own treelet or as an inner node of one further up, which any change further
// down that the root did not see also does), or this pass rewrote a node below.
// Another treelet would find what it found before: the same trees.  Second pass
// over 2M triangles (spheres) 1,930 -> 1,175 us, 280,000 (city) 440 -> 370 us;
// nothing where the first pass rewrote nearly all (heightfield 690 -> 670 us).
//
// Bound by the warp's own chain of steps and, up the tree, by the chain of
// treelets.  A lane's subsets are worked out once and kept in registers (a
// table in constant memory costs a pass per lane), only partitions that hold
// the lowest leaf are formed, and a subset's box is made from its leaves'
// (two 16-byte reads each) so that the table is 1 KB and not 4 per warp.  Two
// passes over 500,000 triangles: 2,854 -> 1,636 us.
constexpr unsigned kWarpAll = 0xFFFFFFFFu;

struct TreeletSmem {
    float4 lo[8], hi[8];  // leaf boxes
    float cost[1 << kTreeletLeaves];
    uint8_t part[1 << kTreeletLeaves];
    int32_t leaf[8], count[8], inner[8];
    int32_t set[8];  // the leaf set of each node of the new treelet
};

// The subsets of 7 leaves by lane: row 0 those of 2 leaves, rows 1-2 of 3 (35
// of them), 3-4 of 4, 5 of 5, and 6 those of 6, each for four lanes; 0 where a
// lane has none.
struct SubsetTable {
    uint8_t set[7][32];
};
constexpr SubsetTable make_subset_table() {
    SubsetTable t{};
    const int first_row[8] = {0, 0, 0, 1, 3, 5, 6, 0};
    int count[8] = {};
    for (int S = 1; S < 128; ++S) {
        int size = 0;
        for (int b = 0; b < 7; ++b) size += (S >> b) & 1;
        if (size < 2 || size > 6) continue;
        const int k = count[size]++;
        if (size == 6) {
            for (int q = 0; q < 4; ++q) t.set[6][4 * k + q] = (uint8_t)S;
        } else {
            t.set[first_row[size] + k / 32][k % 32] = (uint8_t)S;
        }
    }
    return t;
}
__device__ const SubsetTable d_subsets = make_subset_table();

// A lane's subsets: of 2, 3 (two), 4 (two), 5 and 6 leaves; 0 where it has none.
struct LaneSubsets {
    int s2, s3[2], s4[2], s5, s6;
};

// The bits of v deposited into the set bits of R.
__device__ inline int deposit(int v, int R) {
    int Q = 0;
    for (int r = R, b = 0; r; r &= r - 1, ++b)
        if (v & (1 << b)) Q |= r & -r;
    return Q;
}

template <int SIZE>
__device__ inline float subset_area(const TreeletSmem& t, int S) {
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
    for (int i = 0; i < SIZE; ++i, S &= S - 1) {
        const int q = __ffs(S) - 1;
        const float4 l = t.lo[q], h = t.hi[q];
        lo[0] = fminf(lo[0], l.x); lo[1] = fminf(lo[1], l.y); lo[2] = fminf(lo[2], l.z);
        hi[0] = fmaxf(hi[0], h.x); hi[1] = fmaxf(hi[1], h.y); hi[2] = fmaxf(hi[2], h.z);
    }
    return half_area(lo, hi);
}

// The first minimum of COUNT of a subset's partitions, from Q (the part of P
// besides the lowest leaf) down; the last `skip` of them do not count.
template <int COUNT>
__device__ inline void best_partition(const TreeletSmem& t, int S, int Q, int skip, float& bc, int& bp) {
    const int low = S & -S, R = S ^ low;
    bc = FLT_MAX;
    bp = 0;
#pragma unroll 4
    for (int i = 0; i < COUNT; ++i) {
        const int P = low | Q;
        const float c = __fadd_rn(t.cost[P], t.cost[S ^ P]);
        if (c < bc && i < COUNT - skip) { bc = c; bp = P; }
        Q = (Q - 1) & R;
    }
}

template <int SIZE>
__device__ inline void cost_subset(TreeletSmem& t, int S) {
    if (S == 0) return;
    const int R = S & (S - 1);
    float bc;
    int bp;
    best_partition<(1 << (SIZE - 1)) - 1>(t, S, (R - 1) & R, 0, bc, bp);
    t.cost[S] = __fadd_rn(__fmul_rn(kCt, subset_area<SIZE>(t, S)), bc);
    t.part[S] = (uint8_t)bp;
}

// The whole warp restructures the treelet rooted at `root` (warp-uniform),
// which lane `src` has read: its children and their boxes.
__device__ void restructure_warp(BNode* nodes, const NodeBox* leaves, int32_t* leaf_parent, int32_t root,
                                 float root_cost, unsigned stamps, int src, const int2& src_links, const NodeBox& src_left,
                                 const NodeBox& src_right, TreeletSmem& t, const LaneSubsets& mine) {
    const unsigned lane = threadIdx.x & 31u;
    // Grow the treelet: lane q holds leaf q.
    int32_t my_leaf = -1;
    int2 links = make_int2(0, 0);
    NodeBox box{};
    unsigned key = 0u;  // orders the leaves that are nodes by area
    auto take = [&](int32_t code, const NodeBox* known) {
        my_leaf = code;
        if (code >= 0) links = __ldcg(reinterpret_cast<const int2*>(&nodes[code].left));
        if (known) box = *known;
        else box = child_box(nodes, leaves, code);
        const float area = half_area(box.lo, box.hi);
        key = code >= 0 && area > -1.f ? (__float_as_uint(area) & 0x7FFFFFFFu) + 1u : 0u;
    };
    {
        NodeBox l, r;
        for (int a = 0; a < 3; ++a) {
            l.lo[a] = __shfl_sync(kWarpAll, src_left.lo[a], src);
            l.hi[a] = __shfl_sync(kWarpAll, src_left.hi[a], src);
            r.lo[a] = __shfl_sync(kWarpAll, src_right.lo[a], src);
            r.hi[a] = __shfl_sync(kWarpAll, src_right.hi[a], src);
        }
        l.cost = __shfl_sync(kWarpAll, src_left.cost, src);
        l.count = __shfl_sync(kWarpAll, src_left.count, src);
        r.cost = __shfl_sync(kWarpAll, src_right.cost, src);
        r.count = __shfl_sync(kWarpAll, src_right.count, src);
        const int32_t lc = __shfl_sync(kWarpAll, src_links.x, src), rc = __shfl_sync(kWarpAll, src_links.y, src);
        if (lane == 1) l = r;
        if (lane < 2) take(lane == 0 ? lc : rc, &l);
    }
    int n_leaf = 2;
    int my_inner = root;  // lane q: the q-th node of the treelet
    while (n_leaf < kTreeletLeaves) {
        // the first leaf of the largest area that is a node (restructure()'s scan)
        const unsigned most = __reduce_max_sync(kWarpAll, key);
        if (most == 0u) break;
        const int best = __ffs(__ballot_sync(kWarpAll, key == most)) - 1;
        const int32_t x = __shfl_sync(kWarpAll, my_leaf, best);
        const int32_t l = __shfl_sync(kWarpAll, links.x, best), r = __shfl_sync(kWarpAll, links.y, best);
        if ((int)lane == n_leaf - 1) my_inner = x;
        if ((int)lane == best || (int)lane == n_leaf) take((int)lane == best ? l : r, nullptr);
        ++n_leaf;
    }
    if (n_leaf < 3) return;
    if ((int)lane < n_leaf) {
        t.lo[lane] = make_float4(box.lo[0], box.lo[1], box.lo[2], 0.f);
        t.hi[lane] = make_float4(box.hi[0], box.hi[1], box.hi[2], 0.f);
        t.count[lane] = box.count;
        t.leaf[lane] = my_leaf;
        t.inner[lane] = my_inner;
        t.cost[1 << lane] = box.cost;
    }
    __syncwarp();
    const int full = (1 << n_leaf) - 1;
    auto in = [&](int S) { return S <= full ? S : 0; };
    cost_subset<2>(t, in(mine.s2));
    __syncwarp();
    cost_subset<3>(t, in(mine.s3[0]));
    cost_subset<3>(t, in(mine.s3[1]));
    __syncwarp();
    cost_subset<4>(t, in(mine.s4[0]));
    cost_subset<4>(t, in(mine.s4[1]));
    __syncwarp();
    cost_subset<5>(t, in(mine.s5));
    __syncwarp();
    {
        // 6 leaves: 31 partitions over four lanes, eight each in order
        const int S = in(mine.s6), R = S & (S - 1), chunk = (int)(lane & 3u);
        float bc = FLT_MAX;
        int bp = 0, at = chunk;
        if (S) best_partition<8>(t, S, deposit(30 - 8 * chunk, R), chunk == 3 ? 1 : 0, bc, bp);
        for (int o = 2; o > 0; o >>= 1) {
            const float c2 = __shfl_xor_sync(kWarpAll, bc, o);
            const int p2 = __shfl_xor_sync(kWarpAll, bp, o), a2 = __shfl_xor_sync(kWarpAll, at, o);
            if (c2 < bc || (c2 == bc && a2 < at)) { bc = c2; bp = p2; at = a2; }
        }
        if (S && chunk == 0) {
            t.cost[S] = __fadd_rn(__fmul_rn(kCt, subset_area<6>(t, S)), bc);
            t.part[S] = (uint8_t)bp;
        }
    }
    __syncwarp();
    float new_cost;
    if (n_leaf == kTreeletLeaves) {
        // 7 leaves: 63 partitions, two per lane
        const int S = full, R = S ^ 1;
        float bc = FLT_MAX;
        int bp = 0, at = 64;
        for (int i = (int)lane; i < 63; i += 32) {
            const int P = 1 | (((62 - i) << 1) & R);  // R's bits are 1..6: the deposit is a shift
            const float c = __fadd_rn(t.cost[P], t.cost[S ^ P]);
            if (c < bc) { bc = c; bp = P; at = i; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float c2 = __shfl_xor_sync(kWarpAll, bc, o);
            const int p2 = __shfl_xor_sync(kWarpAll, bp, o), a2 = __shfl_xor_sync(kWarpAll, at, o);
            if (c2 < bc || (c2 == bc && a2 < at)) { bc = c2; bp = p2; at = a2; }
        }
        new_cost = __fadd_rn(__fmul_rn(kCt, subset_area<7>(t, S)), bc);
        if (lane == 0) {
            t.cost[S] = new_cost;
            t.part[S] = (uint8_t)bp;
        }
        __syncwarp();
    } else {
        new_cost = t.cost[full];
    }
    if (!(new_cost < 0.999f * root_cost)) return;
    // The new treelet, breadth first: node k has leaf set set[k] and becomes
    // inner[k].  Every set it splits must have a split (finite costs); checked
    // before anything is written.
    bool ok = true;
    if (lane == 0) {
        int n = 1;
        t.set[0] = full;
        for (int q = 0; q < n && ok; ++q) {
            const int S = t.set[q], P = t.part[S];
            if (P == 0 || (P & ~S) != 0 || P == S) { ok = false; break; }
            for (int side = 0; side < 2; ++side) {
                const int T = side ? S ^ P : P;
                if ((T & (T - 1)) == 0) continue;
                if (n >= n_leaf - 1) { ok = false; break; }
                t.set[n++] = T;
            }
        }
        ok = ok && n == n_leaf - 1;
    }
    if (!__shfl_sync(kWarpAll, (int)ok, 0)) return;
    __syncwarp();
    if ((int)lane < n_leaf - 1) {
        const int S = t.set[lane], P = t.part[S];
        const int32_t nd = t.inner[lane];
        int32_t code[2];
        for (int side = 0; side < 2; ++side) {
            const int T = side ? S ^ P : P;
            if ((T & (T - 1)) == 0) {
                code[side] = t.leaf[__ffs(T) - 1];
                if (code[side] >= 0) nodes[code[side]].parent = nd;
                else leaf_parent[~code[side]] = nd;
            } else {
                int q = (int)lane + 1;
                while (q < n_leaf - 2 && t.set[q] != T) ++q;
                code[side] = t.inner[q];
                nodes[t.inner[q]].parent = nd;
            }
        }
        *reinterpret_cast<int2*>(&nodes[nd].left) = make_int2(code[0], code[1]);
        nodes[nd].stamps = stamps;
        NodeBox nb;
        for (int a = 0; a < 3; ++a) { nb.lo[a] = FLT_MAX; nb.hi[a] = -FLT_MAX; }
        nb.count = 0;
        for (int r = S; r; r &= r - 1) {
            const int q = __ffs(r) - 1;
            const float4 l = t.lo[q], h = t.hi[q];
            nb.lo[0] = fminf(nb.lo[0], l.x); nb.lo[1] = fminf(nb.lo[1], l.y); nb.lo[2] = fminf(nb.lo[2], l.z);
            nb.hi[0] = fmaxf(nb.hi[0], h.x); nb.hi[1] = fmaxf(nb.hi[1], h.y); nb.hi[2] = fmaxf(nb.hi[2], h.z);
            nb.count += t.count[q];
        }
        nb.cost = t.cost[S];
        store_box(&nodes[nd].b, nb);
        __threadfence();
    }
    __syncwarp();
}

constexpr int kTreeletWarpBlock = 128;

__global__ void __launch_bounds__(kTreeletWarpBlock, 8) treelet_warp_kernel(
        int64_t n, const NodeBox* leaves, BNode* nodes, int32_t* leaf_parent, int32_t* arrivals, int min_count,
        unsigned pass) {
    __shared__ TreeletSmem smem[kTreeletWarpBlock / 32];
    TreeletSmem& t = smem[threadIdx.x / 32];
    const unsigned lane = threadIdx.x & 31u;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    LaneSubsets mine;
    mine.s2 = d_subsets.set[0][lane];
    mine.s3[0] = d_subsets.set[1][lane];
    mine.s3[1] = d_subsets.set[2][lane];
    mine.s4[0] = d_subsets.set[3][lane];
    mine.s4[1] = d_subsets.set[4][lane];
    mine.s5 = d_subsets.set[5][lane];
    mine.s6 = d_subsets.set[6][lane];
    int32_t node = p < n ? leaf_parent[p] : -1;
    for (;;) {
        bool go = node >= 0;
        if (go) {
            __threadfence();
            if (atomicAdd(&arrivals[node], 1) == 0) go = false;  // the sibling's thread finishes this node
            __threadfence();
        }
        if (!go) node = -1;
        float cost = 0.f;
        bool due = false;
        int32_t parent = -1;  // read ahead of the treelet: only treelets further up change it
        int2 links = make_int2(0, 0);
        NodeBox left{}, right{};
        if (go) {
            const int4 nd = __ldcg(reinterpret_cast<const int4*>(&nodes[node]));
            links = make_int2(nd.x, nd.y);
            parent = nd.z;
            left = child_box(nodes, leaves, links.x);
            right = child_box(nodes, leaves, links.y);
            const NodeBox b = join(left, right);
            cost = b.cost;
            __stcg(&nodes[node].b.cost, cost);
            const bool below = (links.x >= 0 && __ldcg(&nodes[links.x].stamps) >> 16 == pass) ||
                               (links.y >= 0 && __ldcg(&nodes[links.y].stamps) >> 16 == pass);
            const unsigned own = (unsigned)nd.w & 0xFFFFu;
            due = b.count >= min_count && (pass == 1u || own == pass - 1u || below);
            // a treelet that is rewritten stamps its nodes itself
            if (below) __stcg(&nodes[node].stamps, own | (pass << 16));
        }
        unsigned want = __ballot_sync(kWarpAll, due);
        while (want) {
            const int src = __ffs(want) - 1;
            want &= want - 1;
            const int32_t root = __shfl_sync(kWarpAll, node, src);
            const float rc = __shfl_sync(kWarpAll, cost, src);
            restructure_warp(nodes, leaves, leaf_parent, root, rc, pass | (pass << 16), src, links, left, right, t, mine);
        }
        if (go) node = parent;
        if (__ballot_sync(kWarpAll, node >= 0) == 0u) break;
    }
}

// ---- Woop rows (the host woopify, with every rounding explicit so that the
// device gives the host's values for the same triangle).
__device__ void woopify_dev(float3 v0, float3 v1, float3 v2, float4* out) {
    const float3 e0 = make_float3(__fsub_rn(v0.x, v2.x), __fsub_rn(v0.y, v2.y), __fsub_rn(v0.z, v2.z));
    const float3 e1 = make_float3(__fsub_rn(v1.x, v2.x), __fsub_rn(v1.y, v2.y), __fsub_rn(v1.z, v2.z));
    const float3 nn = make_float3(__fsub_rn(__fmul_rn(e0.y, e1.z), __fmul_rn(e0.z, e1.y)),
                                  __fsub_rn(__fmul_rn(e0.z, e1.x), __fmul_rn(e0.x, e1.z)),
                                  __fsub_rn(__fmul_rn(e0.x, e1.y), __fmul_rn(e0.y, e1.x)));
    const double a[3][3] = {{e0.x, e1.x, nn.x}, {e0.y, e1.y, nn.y}, {e0.z, e1.z, nn.z}};
    const double t[3] = {v2.x, v2.y, v2.z};
    auto m2 = [](double p, double q, double r, double s) { return __dsub_rn(__dmul_rn(p, q), __dmul_rn(r, s)); };
    double c[3][3];
    c[0][0] = m2(a[1][1], a[2][2], a[1][2], a[2][1]);
    c[0][1] = m2(a[0][2], a[2][1], a[0][1], a[2][2]);
    c[0][2] = m2(a[0][1], a[1][2], a[0][2], a[1][1]);
    c[1][0] = m2(a[1][2], a[2][0], a[1][0], a[2][2]);
    c[1][1] = m2(a[0][0], a[2][2], a[0][2], a[2][0]);
    c[1][2] = m2(a[0][2], a[1][0], a[0][0], a[1][2]);
    c[2][0] = m2(a[1][0], a[2][1], a[1][1], a[2][0]);
    c[2][1] = m2(a[0][1], a[2][0], a[0][0], a[2][1]);
    c[2][2] = m2(a[0][0], a[1][1], a[0][1], a[1][0]);
    const double det = __dadd_rn(__dadd_rn(__dmul_rn(a[0][0], c[0][0]), __dmul_rn(a[0][1], c[1][0])),
                                 __dmul_rn(a[0][2], c[2][0]));
    if (det == 0.0 || !isfinite(det)) {
        out[0] = out[1] = out[2] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const double rdet = __ddiv_rn(1.0, det);
    double inv[3][4];
    for (int r = 0; r < 3; ++r) {
        for (int q = 0; q < 3; ++q) inv[r][q] = __dmul_rn(c[r][q], rdet);
        inv[r][3] = -__dadd_rn(__dadd_rn(__dmul_rn(inv[r][0], t[0]), __dmul_rn(inv[r][1], t[1])),
                               __dmul_rn(inv[r][2], t[2]));
    }
    float x0 = (float)inv[2][0];
    if (x0 == 0.0f) x0 = 0.0f;  // -0.0f would read as a BVH2 leaf terminator
    out[0] = make_float4(x0, (float)inv[2][1], (float)inv[2][2], (float)(-inv[2][3]));
    out[1] = make_float4((float)inv[0][0], (float)inv[0][1], (float)inv[0][2], (float)inv[0][3]);
    out[2] = make_float4((float)inv[1][0], (float)inv[1][1], (float)inv[1][2], (float)inv[1][3]);
}

struct Item {
    int32_t code;  // binary node (>= 0) or a single-triangle root (< 0)
    int32_t addr;  // 8-wide node index
};

// Counters of the expansion.  alloc[L]: 8-wide nodes of level L in the low
// word, triangle slots taken by level L - 1 in the high word (one atomic takes
// both); node_base[L] / tri_base[L]: nodes / triangle slots of the levels before.
constexpr int kMaxLevels = 4096;
struct Levels {
    unsigned long long alloc[kMaxLevels + 1];
    unsigned int node_base[kMaxLevels + 1];
    unsigned int tri_base[kMaxLevels + 1];
    unsigned int error;
};

// ---- Cost-optimal collapse into 8-wide nodes (the host builder's dynamic
// programme): for every binary node and k = 1..8 slots, the least
// surface-area cost of representing its subtree with at most k children of
// an 8-wide node -- one leaf (at most 3 triangles), an 8-wide node of its
// own, or the node opened with j slots to its left child and k - j to its
// right.  Computed bottom-up (the second child to finish completes a node);
// the expansion then replays the choices instead of opening the largest
// child greedily.
constexpr float kCollapseNode = 1.0f;  // per 8-wide node, times its area
constexpr float kCollapseLeaf = 0.3f;  // per triangle in a leaf, times the leaf's area

struct __align__(16) CollapseDP {
    float best[8];    // k = 1..8
    uint8_t how[8];   // 0 leaf, 1 own node, 2 + j opened with j slots to the left child
    uint8_t split8;   // slots to the left child when the node is an 8-wide node of its own
    uint8_t pad[7];
};

__global__ void collapse_dp_kernel(int64_t n, const NodeBox* leaves, const BNode* nodes, const int32_t* leaf_parent,
                                   int32_t* arrivals, CollapseDP* dp) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int32_t node = leaf_parent[p];
    while (node >= 0) {
        __threadfence();
        if (atomicAdd(&arrivals[node], 1) == 0) return;  // the sibling finishes this node
        __threadfence();
        const int32_t c[2] = {__ldcg(&nodes[node].left), __ldcg(&nodes[node].right)};
        float cost[2][9];
        int32_t prims = 0;
        for (int q = 0; q < 2; ++q) {
            const NodeBox b = child_box(nodes, leaves, c[q]);
            prims += b.count;
            if (c[q] >= 0) {
                const float4* best = reinterpret_cast<const float4*>(dp[c[q]].best);
                const float4 x = __ldcg(best), y = __ldcg(best + 1);
                cost[q][1] = x.x; cost[q][2] = x.y; cost[q][3] = x.z; cost[q][4] = x.w;
                cost[q][5] = y.x; cost[q][6] = y.y; cost[q][7] = y.z; cost[q][8] = y.w;
            } else {
                for (int kk = 1; kk <= 8; ++kk) cost[q][kk] = kCollapseLeaf * half_area(b.lo, b.hi);
            }
        }
        const NodeBox own = child_box(nodes, leaves, node);
        const float av = half_area(own.lo, own.hi);
        float open[9];
        uint8_t split[9];
        for (int kk = 2; kk <= 8; ++kk) {
            open[kk] = FLT_MAX;
            split[kk] = 1;
            for (int j = 1; j < kk; ++j) {
                const float cc = cost[0][j] + cost[1][kk - j];
                if (cc < open[kk]) { open[kk] = cc; split[kk] = (uint8_t)j; }
            }
        }
        CollapseDP d;
        const float as_node = kCollapseNode * av + open[8];
        const float as_leaf = prims <= 3 ? kCollapseLeaf * av * (float)prims : FLT_MAX;
        d.best[0] = fminf(as_leaf, as_node);
        d.how[0] = as_leaf <= as_node ? 0 : 1;
        for (int kk = 2; kk <= 8; ++kk) {
            d.best[kk - 1] = d.best[kk - 2];
            d.how[kk - 1] = d.how[kk - 2];
            if (open[kk] < d.best[kk - 1]) { d.best[kk - 1] = open[kk]; d.how[kk - 1] = (uint8_t)(2 + split[kk]); }
        }
        d.split8 = split[8];
        dp[node] = d;
        node = __ldcg(&nodes[node].parent);
    }
}

// Expands the binary nodes of one level into 8-wide nodes, their slots as the
// collapse chose them.  Eight lanes to a node, one per child: a thread per
// node spent 200-400 us on a level of any size, a chain of a few thousand
// dependent loads and steps with 6 of 32 lanes at work.  A binary node that
// fills k slots owns k neighbouring lanes; opening it hands its right part to
// the lane where that part begins, so children come out in depth-first order
// without a stack, and sums, votes and minima run over the eight lanes.  The
// level's item count is read on the device, so the host queues levels ahead.
// 10 levels of a 500,000-triangle heightfield: 2,204 -> 155 us
// (with eight levels queued past the last).
constexpr int kExpandBlock = 128;

__global__ void __launch_bounds__(kExpandBlock) expand_kernel(
        int level, const Item* items, Item* next, const BNode* nodes, const NodeBox* leaves, const uint64_t* k,
        uint64_t idx_mask, const int32_t* ref_tri, float4* out_nodes, unsigned node_cap, int32_t* prim,
        unsigned tri_cap, Levels* lv, const CollapseDP* dp) {
    constexpr int kGroups = kExpandBlock / 8;
    __shared__ float4 node_smem[kGroups][5];
    __shared__ int32_t open_code[kGroups][8];
    __shared__ int open_slots[kGroups][8];
    const unsigned lane = threadIdx.x & 31u, shift = lane & 24u;
    const int c = (int)(lane & 7u), group = (int)(threadIdx.x >> 3);
    // Levels queued behind one that failed have nothing valid to read.
    if (lv->error) return;
    // Where this level's triangles and the next one's nodes begin: after all
    // that the levels before took.
    const unsigned n_items = (unsigned)lv->alloc[level];
    const unsigned next0 = lv->node_base[level] + n_items;
    const unsigned tri0 = level ? lv->tri_base[level - 1] + (unsigned)(lv->alloc[level] >> 32) : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        lv->node_base[level + 1] = next0;
        lv->tri_base[level] = tri0;
    }
    auto octet = [&](bool b) -> unsigned { return (__ballot_sync(kWarpAll, b) >> shift) & 0xFFu; };
    auto all_or = [&](unsigned x) -> unsigned {
        for (int m = 4; m > 0; m >>= 1) x |= __shfl_xor_sync(kWarpAll, x, m);
        return x;
    };
    const unsigned groups = gridDim.x * kGroups;
    // warp-uniform loop: the groups of a warp take neighbouring items
    for (unsigned w0 = blockIdx.x * kGroups + (threadIdx.x >> 5) * 4; w0 < n_items; w0 += groups) {
        const unsigned w = w0 + (shift >> 3);
        const bool active = w < n_items;
        unsigned err = 0u;
        Item it{0, 0};
        if (active) it = items[w];
        // ---- the children: lane q holds the binary node whose slots begin at q
        bool has = false;
        int32_t code = 0;
        int slots = 0;
        if (active) {
            if (it.code < 0) {  // one triangle: the root holds one leaf
                has = c == 0;
                code = it.code;
                slots = 8;
            } else {
                const int s8 = dp[it.code].split8;
                const int2 lr = *reinterpret_cast<const int2*>(&nodes[it.code].left);
                if (s8 < 1 || s8 > 7) {
                    err = 4u;
                } else if (c == 0) {
                    has = true;
                    code = lr.x;
                    slots = s8;
                } else if (c == s8) {
                    has = true;
                    code = lr.y;
                    slots = 8 - s8;
                }
            }
        }
        for (int step = 0; step < 8; ++step) {
            const int how = has && code >= 0 && slots >= 1 ? dp[code].how[slots - 1] : 0;
            bool open = how >= 2;
            const int j = how - 2;
            if (open && (j < 1 || j >= slots || step == 7)) {  // a table that opens more than it has slots
                err = 4u;
                open = false;
            }
            if (!__any_sync(kWarpAll, open)) break;
            open_slots[group][c] = 0;
            __syncwarp();
            if (open) {
                const int2 lr = *reinterpret_cast<const int2*>(&nodes[code].left);
                open_code[group][c + j] = lr.y;
                open_slots[group][c + j] = slots - j;
                code = lr.x;
                slots = j;
            }
            __syncwarp();
            if (open_slots[group][c]) {
                has = true;
                code = open_code[group][c];
                slots = open_slots[group][c];
            }
            __syncwarp();
        }
        NodeBox b{};
        if (has) b = child_box(nodes, leaves, code);
        // ---- node box
        float lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = has ? b.lo[a] : FLT_MAX;
            hi[a] = has ? b.hi[a] : -FLT_MAX;
            for (int m = 4; m > 0; m >>= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(kWarpAll, lo[a], m));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(kWarpAll, hi[a], m));
            }
        }
        // ---- octant slots: cheapest (slot, child) pairs first, as the host
        // converter; equal costs to the lower slot, then the lower child
        float nc[3], cc[3];
        for (int a = 0; a < 3; ++a) {
            nc[a] = (lo[a] + hi[a]) * 0.5f;
            cc[a] = __fsub_rn(__fmul_rn(__fadd_rn(b.lo[a], b.hi[a]), 0.5f), nc[a]);
        }
        int my_slot = -1;
        unsigned free_slots = 0xFFu;
        for (int round = 0; round < 8; ++round) {
            float best = FLT_MAX;
            int who = 64;  // slot * 8 + lane
            if (has && my_slot < 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float cost = __fadd_rn(__fadd_rn((q & 4) ? -cc[0] : cc[0], (q & 2) ? -cc[1] : cc[1]),
                                                 (q & 1) ? -cc[2] : cc[2]);
                    if (((free_slots >> q) & 1u) && cost < best) {
                        best = cost;
                        who = q * 8 + c;
                    }
                }
            }
            for (int m = 4; m > 0; m >>= 1) {
                const float b2 = __shfl_xor_sync(kWarpAll, best, m);
                const int w2 = __shfl_xor_sync(kWarpAll, who, m);
                if (b2 < best || (b2 == best && w2 < who)) {
                    best = b2;
                    who = w2;
                }
            }
            if (who < 64) {
                free_slots &= ~(1u << (who >> 3));
                if ((who & 7) == c) my_slot = who >> 3;
            }
            if (!__any_sync(kWarpAll, who < 64)) break;
        }
        // Costs that are not below FLT_MAX (infinite or NaN vertices, centres
        // that overflow) choose nothing: those children take the free slots in
        // order, since every inner child's place in the queue will be read.
        const unsigned unplaced = octet(has && my_slot < 0);
        if (has && my_slot < 0) {
            unsigned f = free_slots;
            for (int rank = __popc(unplaced & ((1u << c) - 1u)); rank > 0; --rank) f &= f - 1u;
            my_slot = __ffs(f) - 1;
        }
        // ---- per-axis exponent, grown while a child's upper bound does not fit a byte
        int e[3];
        for (int a = 0; a < 3; ++a) {
            const float r = ceilf(log2f((hi[a] - lo[a]) / 255.0f));
            e[a] = isfinite(r) ? (int)fmaxf(-127.f, fminf(127.f, r)) : 0;
            for (;;) {
                const float scale = ldexpf(1.0f, e[a]);
                const bool over = has && (int)ceilf((b.hi[a] - lo[a]) / scale) > 255;
                const bool grow = octet(over) != 0u && e[a] < 127;
                if (grow) ++e[a];
                if (!__any_sync(kWarpAll, grow)) break;
            }
        }
        // ---- allocations: inner children as one block, leaf triangles as one
        // run, taken for the warp's four nodes by one atomic
        const bool inner = has && b.count > 3, leaf = has && !inner;
        const unsigned n_inner = __popc(octet(inner));
        unsigned n_tris = leaf ? (unsigned)b.count : 0u;
        for (int m = 4; m > 0; m >>= 1) n_tris += __shfl_xor_sync(kWarpAll, n_tris, m);
        const unsigned long long want = ((unsigned long long)n_tris << 32) | n_inner;
        unsigned long long before = 0ull, total = 0ull;
        for (int q = 0; q < 4; ++q) {
            const unsigned long long x = __shfl_sync(kWarpAll, want, 8 * q);
            if (q < (int)(shift >> 3)) before += x;
            total += x;
        }
        unsigned long long got = 0ull;
        if (lane == 0 && total) got = atomicAdd(&lv->alloc[level + 1], total);
        got = __shfl_sync(kWarpAll, got, 0) + before;
        const unsigned qbase = (unsigned)got;
        const unsigned base = next0 + qbase, tbase = tri0 + (unsigned)(got >> 32);
        if (active && !err && ((uint64_t)base + n_inner > node_cap || (uint64_t)tbase + n_tris > tri_cap)) err = 1u;
        err = all_or(err);  // of the group
        const bool go = active && err == 0u;
        // ---- the node
        const unsigned imask = all_or(inner ? 1u << my_slot : 0u);
        const unsigned counts = all_or(leaf ? (unsigned)b.count << (2 * my_slot) : 0u);
        const unsigned below = has ? counts & ((1u << (2 * my_slot)) - 1u) : 0u;
        const unsigned first_tri = __popc(below & 0x5555u) + 2u * __popc(below & 0xAAAAu);
        const unsigned all_tris = __popc(counts & 0x5555u) + 2u * __popc(counts & 0xAAAAu);
        if (c < 5) node_smem[group][c] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        unsigned char* bytes = reinterpret_cast<unsigned char*>(node_smem[group]);
        if (go && c == 0) {
            node_smem[group][0] = make_float4(lo[0], lo[1], lo[2],
                                              __uint_as_float(((unsigned)e[0] & 0xFFu) | (((unsigned)e[1] & 0xFFu) << 8) |
                                                              (((unsigned)e[2] & 0xFFu) << 16) | (imask << 24)));
            reinterpret_cast<uint2*>(bytes)[2] = make_uint2(imask ? base : 0u, all_tris ? tbase : 0u);
        }
        if (go && has) {
            for (int a = 0; a < 3; ++a) {
                const float scale = ldexpf(1.0f, e[a]);
                bytes[32 + my_slot + 8 * a] = (uint8_t)(int)floorf((b.lo[a] - lo[a]) / scale);
                bytes[32 + my_slot + 8 * (3 + a)] = (uint8_t)(int)ceilf((b.hi[a] - lo[a]) / scale);
            }
            if (inner) {
                const unsigned rank = __popc(imask & ((1u << my_slot) - 1u));
                bytes[24 + my_slot] = (uint8_t)((1u << 5) | (24u + my_slot));
                next[qbase + rank] = Item{code, (int32_t)(base + rank)};
            } else {
                const uint32_t unary = b.count == 1 ? 1u : (b.count == 2 ? 3u : 7u);
                bytes[24 + my_slot] = (uint8_t)((unary << 5) | (first_tri & 31u));
                // the child's triangles, left first: a leaf, or a subtree of at most 3
                int32_t st[4];
                int sp = 0;
                unsigned t = 0;
                st[sp++] = code;
                while (sp > 0) {
                    const int32_t x = st[--sp];
                    if (t >= (unsigned)b.count || (x >= 0 && sp + 2 > 4)) {  // counts disagree with the tree
                        err = 2u;
                        break;
                    }
                    if (x < 0) {
                        const int64_t ref = key_tri(k, ~x, idx_mask);
                        const int64_t slot = 3 * ((int64_t)tbase + first_tri + t);
                        prim[slot] = ref_tri ? ref_tri[ref] : (int32_t)ref;
                        ++t;
                    } else {
                        st[sp++] = nodes[x].right;
                        st[sp++] = nodes[x].left;
                    }
                }
            }
        }
        __syncwarp();
        if (go && c < 5) out_nodes[(int64_t)it.addr * 5 + c] = node_smem[group][c];
        if (err) atomicOr(&lv->error, err);
        __syncwarp();
    }
}

// Woop rows of the stored triangles, a thread each (prim: the triangle of
// each slot's first row, -1 in a slot nothing took).
__global__ void woop_rows_kernel(int64_t n, const float* v, const int32_t* idx, float4* woop, const int32_t* prim) {
    const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const int32_t tri = prim[3 * slot];
    if (tri < 0) {
        woop[3 * slot] = woop[3 * slot + 1] = woop[3 * slot + 2] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const int32_t* ti = idx + 3 * (int64_t)tri;
    float4 rows[3];
    woopify_dev(vtx(v, ti[0]), vtx(v, ti[1]), vtx(v, ti[2]), rows);
    for (int q = 0; q < 3; ++q) woop[3 * slot + q] = rows[q];
}

unsigned blocks_of(int64_t n, int b) { return (unsigned)std::max<int64_t>(1, (n + b - 1) / b); }

// ---- PLOC: parallel locally-ordered clustering (Meister and Bittner,
// "Parallel Locally-Ordered Clustering for Bounding Volume Hierarchy
// Construction", IEEE TVCG 2018).  The clusters start as the triangles in
// Morton order; each round every cluster finds, among the kPlocRadius
// clusters on either side of it, the one whose merged box has the least
// surface area, mutual nearest neighbours merge into a new node (placed at
// the lower position), and the array is compacted.  Merged boxes group
// primitives by extent as well as position, which the Morton order alone
// does not.  Node numbers come from prefix sums, counting down from n - 2 in
// position order, so the last merge is the root (node 0) and the tree does
// not depend on thread scheduling.
//
// A round is three launches over tiles of kPlocTile clusters: the nearest
// neighbours of a tile and of the kPlocRadius clusters either side of it (so
// that a tile knows its mutual pairs), with the tile's numbers of merges and
// survivors; one block that sums those over the tiles; and the merge, which
// writes the survivors and merged clusters to the other buffer.  Cluster
// counts stay on the device and rounds are queued ahead of them.  Once
// kPlocLast clusters or fewer are left, most of the rounds but little of the
// work, one block does the remaining rounds in shared memory.  A cluster
// carries its box, cost and count, so a merge reads nothing of the tree.
// 500,000-triangle heightfield, 51 rounds: 1,320 us of kernels with two scans
// and two copies to the host in every round -> 580 us and five copies.
constexpr int kPlocRadius = 16;
constexpr int kPlocTile = 256;
constexpr int kPlocLast = 2048;
constexpr int kPlocRoundsAhead = 6;

struct PlocState {
    int32_t m;      // clusters
    int32_t top;    // next node number (counting down)
    int32_t cur;    // buffer holding the clusters
    uint32_t error; // a round that merged nothing (non-finite boxes)
};
struct Clusters {
    int32_t* code[2];
    NodeBox* box[2];
};

// Nearest neighbour of cluster i within the radius: least merged area, ties
// to the nearer position, then to the cluster's partner i ^ 1, then to the
// lower position.  The rule is the same seen from both sides of a pair, and
// clusters with identical boxes (duplicated geometry) pair off with their
// partners, half of them merging per round instead of one pair.
template <class GetBox>
__device__ inline int ploc_nearest(int i, int m, const NodeBox& bi, GetBox box) {
    const int j0 = i - kPlocRadius < 0 ? 0 : i - kPlocRadius;
    const int j1 = i + kPlocRadius >= m ? m - 1 : i + kPlocRadius;
    float best = FLT_MAX;
    int bj = i == 0 ? 1 : i - 1, bdist = INT32_MAX;
    bool bpartner = false;
    for (int j = j0; j <= j1; ++j) {
        if (j == i) continue;
        float4 l, h;
        box(j, l, h);
        const float lo[3] = {fminf(bi.lo[0], l.x), fminf(bi.lo[1], l.y), fminf(bi.lo[2], l.z)};
        const float hi[3] = {fmaxf(bi.hi[0], h.x), fmaxf(bi.hi[1], h.y), fmaxf(bi.hi[2], h.z)};
        const float d = half_area(lo, hi);
        const int dist = j > i ? j - i : i - j;
        const bool partner = j == (i ^ 1);
        // ascending j: among full ties the first is the lowest position
        if (d < best || (d == best && (dist < bdist || (dist == bdist && partner && !bpartner)))) {
            best = d;
            bj = j;
            bdist = dist;
            bpartner = partner;
        }
    }
    return bj;
}

// A cluster's part in a round.
constexpr uint8_t kPlocMerges = 0x40;    // lower cluster of a mutual pair
constexpr uint8_t kPlocAbsorbed = 0x80;  // upper one; low six bits: neighbour - cluster + kPlocRadius

__global__ void ploc_init_kernel(int64_t n, const NodeBox* leaves, Clusters cl, PlocState* st) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) st[0] = PlocState{(int32_t)n, (int32_t)(n - 2), 0, 0u};
    if (p >= n) return;
    cl.code[0][p] = ~(int32_t)p;
    store_box(&cl.box[0][p], child_box(nullptr, leaves, ~(int32_t)p));
}

__device__ inline bool ploc_idle(const PlocState& s) { return s.error || s.m <= kPlocLast; }

__global__ void __launch_bounds__(kPlocTile + 2 * kPlocRadius) ploc_pairs_kernel(Clusters cl, const PlocState* st,
                                                                                 uint8_t* part, uint2* sums) {
    constexpr int kReach = 2 * kPlocRadius;
    __shared__ float4 slo[kPlocTile + 2 * kReach], shi[kPlocTile + 2 * kReach];
    __shared__ int snn[kPlocTile + 2 * kPlocRadius];
    __shared__ unsigned counts[2];
    const PlocState s = *st;
    const int t0 = blockIdx.x * kPlocTile;
    if (ploc_idle(s) || t0 >= s.m) return;
    const NodeBox* box = cl.box[s.cur];
    for (int q = threadIdx.x; q < kPlocTile + 2 * kReach; q += blockDim.x) {
        const int j = t0 - kReach + q;
        if (j < 0 || j >= s.m) continue;
        const float4* p = reinterpret_cast<const float4*>(box + j);
        slo[q] = p[0];
        shi[q] = p[1];
    }
    if (threadIdx.x < 2) counts[threadIdx.x] = 0u;
    __syncthreads();
    const int i = t0 - kPlocRadius + (int)threadIdx.x;
    int nn = -1;
    if (i >= 0 && i < s.m) {
        const float4 l = slo[threadIdx.x + kPlocRadius], h = shi[threadIdx.x + kPlocRadius];
        NodeBox bi;
        bi.lo[0] = l.x; bi.lo[1] = l.y; bi.lo[2] = l.z;
        bi.hi[0] = h.x; bi.hi[1] = h.y; bi.hi[2] = h.z;
        nn = ploc_nearest(i, s.m, bi, [&](int j, float4& jl, float4& jh) {
            jl = slo[j - t0 + kReach];
            jh = shi[j - t0 + kReach];
        });
    }
    snn[threadIdx.x] = nn;
    __syncthreads();
    bool merges = false, keeps = false;
    if (i >= t0 && i < t0 + kPlocTile && i < s.m) {
        const bool mutual = snn[nn - t0 + kPlocRadius] == i;
        merges = mutual && i < nn;
        const bool absorbed = mutual && i > nn;
        keeps = !absorbed;
        part[i] = (uint8_t)((nn - i + kPlocRadius) | (merges ? kPlocMerges : 0) | (absorbed ? kPlocAbsorbed : 0));
    }
    const unsigned bm = __ballot_sync(kWarpAll, merges), bk = __ballot_sync(kWarpAll, keeps);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&counts[0], (unsigned)__popc(bm));
        atomicAdd(&counts[1], (unsigned)__popc(bk));
    }
    __syncthreads();
    if (threadIdx.x == 0) sums[blockIdx.x] = make_uint2(counts[0], counts[1]);
}

// Exclusive sums of the tiles' counts, and the state of the next round.
__global__ void __launch_bounds__(1024) ploc_scan_kernel(const PlocState* st, PlocState* st_next, uint2* sums) {
    __shared__ uint2 warp_sum[32];
    const PlocState s = *st;
    if (ploc_idle(s)) {
        if (threadIdx.x == 0) *st_next = s;
        return;
    }
    const int tiles = (s.m + kPlocTile - 1) / kPlocTile;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint2 carry = make_uint2(0u, 0u);
    for (int t = 0; t < tiles; t += 1024) {
        const int q = t + (int)threadIdx.x;
        const uint2 own = q < tiles ? sums[q] : make_uint2(0u, 0u);
        uint2 x = own;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned a = __shfl_up_sync(kWarpAll, x.x, o), b = __shfl_up_sync(kWarpAll, x.y, o);
            if (lane >= (unsigned)o) { x.x += a; x.y += b; }
        }
        if (lane == 31u) warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint2 y = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned a = __shfl_up_sync(kWarpAll, y.x, o), b = __shfl_up_sync(kWarpAll, y.y, o);
                if (lane >= (unsigned)o) { y.x += a; y.y += b; }
            }
            warp_sum[lane] = y;
        }
        __syncthreads();
        uint2 before = carry;
        if (warp > 0) { before.x += warp_sum[warp - 1].x; before.y += warp_sum[warp - 1].y; }
        if (q < tiles) sums[q] = make_uint2(before.x + x.x - own.x, before.y + x.y - own.y);
        carry.x += warp_sum[31].x;
        carry.y += warp_sum[31].y;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        PlocState n = s;
        const int32_t merges = (int32_t)carry.x, kept = (int32_t)carry.y;
        if (merges <= 0 || kept != s.m - merges || s.top - merges + 1 < 0) {
            n.error = 1u;
        } else {
            n.m = kept;
            n.top = s.top - merges;
            n.cur = s.cur ^ 1;
        }
        *st_next = n;
    }
}

// A merged pair becomes node `node`.
__device__ inline void ploc_link(BNode* nodes, int32_t node, int32_t left, int32_t right,
                                 const NodeBox& b) {
    *reinterpret_cast<int4*>(&nodes[node]) = make_int4(left, right, -1, 0);
    store_box(&nodes[node].b, b);
}
__device__ inline void ploc_set_parent(BNode* nodes, int32_t* leaf_parent, int32_t code, int32_t node) {
    if (code >= 0) nodes[code].parent = node;
    else leaf_parent[~code] = node;
}

__global__ void __launch_bounds__(kPlocTile) ploc_merge_kernel(Clusters cl, const PlocState* st, const PlocState* st_next,
                                                               const uint8_t* part, const uint2* sums, BNode* nodes,
                                                               int32_t* leaf_parent) {
    __shared__ uint2 warp_sum[kPlocTile / 32];
    const PlocState s = *st;
    const int i = blockIdx.x * kPlocTile + threadIdx.x;
    if (ploc_idle(s) || st_next->error || blockIdx.x * kPlocTile >= s.m) return;
    const uint8_t f = i < s.m ? part[i] : kPlocAbsorbed;
    const bool merges = (f & kPlocMerges) != 0, keeps = (f & kPlocAbsorbed) == 0;
    const unsigned bm = __ballot_sync(kWarpAll, merges), bk = __ballot_sync(kWarpAll, keeps);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    if (lane == 0) warp_sum[warp] = make_uint2(__popc(bm), __popc(bk));
    __syncthreads();
    uint2 at = sums[blockIdx.x];
    for (unsigned q = 0; q < warp; ++q) { at.x += warp_sum[q].x; at.y += warp_sum[q].y; }
    if (!keeps) return;
    const int32_t node = s.top - (int32_t)(at.x + __popc(bm & below));
    const unsigned to = at.y + __popc(bk & below);
    const int32_t* code = cl.code[s.cur];
    const NodeBox* box = cl.box[s.cur];
    int32_t c = code[i];
    NodeBox b = child_box(nullptr, box, ~i);
    if (merges) {
        const int j = i + (int)(f & 0x3Fu) - kPlocRadius;
        const int32_t c2 = code[j];
        b = join(b, child_box(nullptr, box, ~j));
        ploc_link(nodes, node, c, c2, b);
        ploc_set_parent(nodes, leaf_parent, c, node);
        ploc_set_parent(nodes, leaf_parent, c2, node);
        c = node;
    }
    cl.code[s.cur ^ 1][to] = c;
    store_box(&cl.box[s.cur ^ 1][to], b);
}

// All rounds from kPlocLast clusters on, in one block.
struct PlocLast {
    float4 lo[2][kPlocLast], hi[2][kPlocLast];  // lo.w: cost, hi.w: count
    int32_t code[2][kPlocLast];
    int32_t nn[kPlocLast];
    uint2 warp_sum[32];
};

__global__ void __launch_bounds__(1024) ploc_last_kernel(Clusters cl, PlocState* st, BNode* nodes,
                                                         int32_t* leaf_parent) {
    extern __shared__ __align__(16) unsigned char raw[];
    PlocLast& t = *reinterpret_cast<PlocLast*>(raw);
    const PlocState s = *st;
    if (s.error || s.m > kPlocLast) return;
    int m = s.m, top = s.top, cur = 0;
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
        const float4* p = reinterpret_cast<const float4*>(&cl.box[s.cur][q]);
        t.lo[0][q] = p[0];
        t.hi[0][q] = p[1];
        t.code[0][q] = cl.code[s.cur][q];
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    uint32_t error = 0u;
    while (m > 1) {
        auto load = [&](int j, float4& l, float4& h) {
            l = t.lo[cur][j];
            h = t.hi[cur][j];
        };
        auto get = [&](int j) {
            float4 l, h;
            load(j, l, h);
            NodeBox b;
            b.lo[0] = l.x; b.lo[1] = l.y; b.lo[2] = l.z; b.cost = l.w;
            b.hi[0] = h.x; b.hi[1] = h.y; b.hi[2] = h.z; b.count = __float_as_int(h.w);
            return b;
        };
        for (int i = threadIdx.x; i < m; i += blockDim.x) t.nn[i] = ploc_nearest(i, m, get(i), load);
        __syncthreads();
        int merged = 0, kept = 0;
        for (int i0 = 0; i0 < m; i0 += blockDim.x) {
            const int i = i0 + (int)threadIdx.x;
            bool merges = false, keeps = false;
            int j = 0;
            if (i < m) {
                j = t.nn[i];
                const bool mutual = t.nn[j] == i;
                merges = mutual && i < j;
                keeps = !(mutual && i > j);
            }
            const unsigned bm = __ballot_sync(kWarpAll, merges), bk = __ballot_sync(kWarpAll, keeps);
            if (lane == 0) t.warp_sum[warp] = make_uint2(__popc(bm), __popc(bk));
            __syncthreads();
            uint2 x = t.warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned a = __shfl_up_sync(kWarpAll, x.x, o), b = __shfl_up_sync(kWarpAll, x.y, o);
                if (lane >= (unsigned)o) { x.x += a; x.y += b; }
            }
            const unsigned all_m = __shfl_sync(kWarpAll, x.x, 31), all_k = __shfl_sync(kWarpAll, x.y, 31);
            const unsigned wm = __shfl_sync(kWarpAll, x.x, warp ? warp - 1 : 0);
            const unsigned wk = __shfl_sync(kWarpAll, x.y, warp ? warp - 1 : 0);
            if (keeps) {
                const int32_t node = top - (merged + (int)(warp ? wm : 0u) + __popc(bm & below));
                const int to = kept + (int)(warp ? wk : 0u) + __popc(bk & below);
                int32_t c = t.code[cur][i];
                NodeBox b = get(i);
                if (merges && node >= 0) {
                    const int32_t c2 = t.code[cur][j];
                    b = join(b, get(j));
                    ploc_link(nodes, node, c, c2, b);
                    ploc_set_parent(nodes, leaf_parent, c, node);
                    ploc_set_parent(nodes, leaf_parent, c2, node);
                    c = node;
                }
                t.code[cur ^ 1][to] = c;
                t.lo[cur ^ 1][to] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.cost);
                t.hi[cur ^ 1][to] = make_float4(b.hi[0], b.hi[1], b.hi[2], __int_as_float(b.count));
            }
            merged += (int)all_m;
            kept += (int)all_k;
            __syncthreads();
        }
        if (merged <= 0 || kept != m - merged || top - merged + 1 < 0) {  // uniform: every thread has the same sums
            error = 1u;
            break;
        }
        m = kept;
        top -= merged;
        cur ^= 1;
    }
    if (threadIdx.x == 0) *st = PlocState{m, top, s.cur, error};
}

}  // namespace
}  // namespace rq

using namespace rq;

// Where builds take their scratch from: a memory pool per device that keeps
// up to kPoolKeepBytes between builds while a scene built on the device lives
// (a new block of memory costs ~330 us to map and ~270 us to unmap, up to
// several ms now and then; a build of 500,000 triangles takes 4 ms besides).
// The memory goes back to the device with the last such scene, so a caller that
// destroys each scene before it builds the next maps it anew every time (500,000
// triangles 3.6 -> 4.0 ms, and the destruction takes 1.2).  A pool is
// safe for any number of threads and streams, and hands a block that one
// stream freed to another only in order.
constexpr uint64_t kPoolKeepBytes = 256ull << 20;  // the scratch of about a million triangles

struct ScratchPool {
    std::mutex mu;
    struct Device {
        cudaMemPool_t pool = nullptr;
        int users = 0;  // scenes built on the device and builds under way
    };
    std::map<int, Device> devices;

    cudaError_t enter(int dev, cudaMemPool_t* pool) {
        std::lock_guard<std::mutex> lk(mu);
        Device& d = devices[dev];
        if (!d.pool) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaError_t e = cudaMemPoolCreate(&d.pool, &props);
            if (e != cudaSuccess) return e;
            uint64_t keep = kPoolKeepBytes;
            e = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
            if (e != cudaSuccess) {
                cudaMemPoolDestroy(d.pool);
                d.pool = nullptr;
                return e;
            }
        }
        ++d.users;
        *pool = d.pool;
        return cudaSuccess;
    }
    void leave(int dev) {
        std::lock_guard<std::mutex> lk(mu);
        Device& d = devices[dev];
        if (--d.users == 0) cudaMemPoolTrimTo(d.pool, 0);
    }
};
static ScratchPool& scratch_pool() {
    static ScratchPool* p = new ScratchPool();  // never destroyed: scenes may outlive static objects
    return *p;
}
void rq::gpu_built_scene_gone(int device, cudaEvent_t scratch_freed) {
    cudaEventSynchronize(scratch_freed);
    cudaEventDestroy(scratch_freed);
    scratch_pool().leave(device);
}

// One allocation from the pool cut into aligned buffers: laid out first, then
// made.
struct Arena {
    char* base = nullptr;
    size_t bytes = 0;
    cudaStream_t stream = nullptr;
    std::vector<std::pair<void**, size_t>> parts;
    template <class T>
    void add(T** p, int64_t count) {
        parts.emplace_back((void**)p, bytes);
        bytes += ((size_t)std::max<int64_t>(1, count) * sizeof(T) + 255) / 256 * 256;
    }
    cudaError_t make(cudaMemPool_t pool, cudaStream_t s) {
        stream = s;
        const cudaError_t e = cudaMallocFromPoolAsync((void**)&base, std::max<size_t>(bytes, 256), pool, s);
        if (e == cudaSuccess)
            for (auto& p : parts) *p.first = base + p.second;
        return e;
    }
    void release() {
        if (base) cudaFreeAsync(base, stream);
        base = nullptr;
    }
    ~Arena() { release(); }
};

// Buffers of the PLOC rounds.
struct PlocBuffers {
    Clusters cl{};
    uint8_t* part = nullptr;
    uint2* sums = nullptr;
    PlocState* state = nullptr;  // two, by the parity of the round
    void layout(Arena& a, int64_t n) {
        for (int q = 0; q < 2; ++q) {
            a.add(&cl.code[q], n);
            a.add(&cl.box[q], n);
        }
        a.add(&part, n);
        a.add(&sums, (n + kPlocTile - 1) / kPlocTile);
        a.add(&state, 2);
    }
};

// PLOC rounds on the leaves of the sorted triangles: nodes, boxes, counts,
// costs and parent links as the radix tree + bottom-up boxes give them.
static rq_status ploc_tree(const PlocBuffers& p, int64_t n, const NodeBox* leaves, BNode* bn, int32_t* leaf_parent,
                           cudaStream_t s) {
    RQ_CUDA(cudaFuncSetAttribute(ploc_last_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PlocLast)));
    ploc_init_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, leaves, p.cl, p.state);
    RQ_CUDA(cudaGetLastError());
    PlocState now{(int32_t)n, (int32_t)(n - 2), 0, 0u};
    int parity = 0;
    // A round merges at least the globally closest pair in reach (one that
    // merges nothing sets the error), so the clusters run out.
    for (int64_t round = 0; now.m > kPlocLast; round += kPlocRoundsAhead) {
        if (round > 100000) return RQ_ERR_BAD_SCENE;
        const unsigned tiles = blocks_of(now.m, kPlocTile);
        for (int q = 0; q < kPlocRoundsAhead; ++q, parity ^= 1) {
            ploc_pairs_kernel<<<tiles, kPlocTile + 2 * kPlocRadius, 0, s>>>(p.cl, p.state + parity, p.part, p.sums);
            ploc_scan_kernel<<<1, 1024, 0, s>>>(p.state + parity, p.state + (parity ^ 1), p.sums);
            ploc_merge_kernel<<<tiles, kPlocTile, 0, s>>>(p.cl, p.state + parity, p.state + (parity ^ 1), p.part, p.sums,
                                                          bn, leaf_parent);
        }
        RQ_CUDA(cudaGetLastError());
        RQ_CUDA(cudaMemcpyAsync(&now, p.state + parity, sizeof(now), cudaMemcpyDeviceToHost, s));
        RQ_CUDA(cudaStreamSynchronize(s));
        if (now.error) return RQ_ERR_BAD_SCENE;
    }
    ploc_last_kernel<<<1, 1024, sizeof(PlocLast), s>>>(p.cl, p.state + parity, bn, leaf_parent);
    RQ_CUDA(cudaGetLastError());
    RQ_CUDA(cudaMemcpyAsync(&now, p.state + parity, sizeof(now), cudaMemcpyDeviceToHost, s));
    RQ_CUDA(cudaStreamSynchronize(s));
    return now.error || now.m != 1 || now.top != -1 ? RQ_ERR_BAD_SCENE : RQ_OK;  // n - 1 nodes, the root last (node 0)
}

// The references of a pre-split mesh: the box mesh (2 corners per
// reference), its index triples and the triangle of each reference.
struct RefMesh {
    float* v = nullptr;
    int32_t* idx = nullptr;
    int32_t* tri = nullptr;
    int64_t n = 0;
    Arena arena;
};

// Cuts the nt triangles into at most nt + nt * budget / 100 references
// (fewer when few triangles waste box area).  Leaves rm.n = 0 when there is
// nothing to split.  The indices have been checked.
static rq_status presplit(const float* v, const int32_t* idx, int64_t nt, int budget, RefMesh& rm, cudaMemPool_t pool,
                          cudaStream_t s) {
    const int64_t extra = std::min<int64_t>((int64_t)((double)nt * budget / 100.0), (int64_t)INT32_MAX / 4 - nt);
    if (extra <= 0) return RQ_OK;
    unsigned* sb = nullptr;
    float *prio = nullptr, *sum = nullptr;
    int64_t *pieces = nullptr, *off = nullptr;
    char* temp = nullptr;
    size_t b_sum = 0, b_scan = 0;
    RQ_CUDA(cub::DeviceReduce::Sum(nullptr, b_sum, prio, sum, (int)nt, s));
    RQ_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b_scan, pieces, off, (int)nt, s));
    Arena arena;  // freed in stream order, after the kernels that read it
    arena.add(&sb, 6);
    arena.add(&prio, nt);
    arena.add(&sum, 1);
    arena.add(&pieces, nt);
    arena.add(&off, nt);
    arena.add(&temp, (int64_t)std::max(b_sum, b_scan));
    RQ_CUDA(arena.make(pool, s));
    const unsigned init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    RQ_CUDA(cudaMemcpyAsync(sb, init, sizeof(init), cudaMemcpyHostToDevice, s));
    scene_bounds_kernel<<<std::min<unsigned>(blocks_of(nt, 256), 4 * 148), 256, 0, s>>>(v, idx, nt, sb);
    split_priority_kernel<<<blocks_of(nt, 256), 256, 0, s>>>(v, idx, nt, sb, prio);
    RQ_CUDA(cudaGetLastError());
    RQ_CUDA(cub::DeviceReduce::Sum(temp, b_sum, prio, sum, (int)nt, s));
    split_count_kernel<<<blocks_of(nt, 256), 256, 0, s>>>(prio, nt, sum, (double)extra, pieces);
    RQ_CUDA(cudaGetLastError());
    RQ_CUDA(cub::DeviceScan::ExclusiveSum(temp, b_scan, pieces, off, (int)nt, s));
    int64_t tail[2] = {0, 0};
    RQ_CUDA(cudaMemcpyAsync(&tail[0], off + nt - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RQ_CUDA(cudaMemcpyAsync(&tail[1], pieces + nt - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RQ_CUDA(cudaStreamSynchronize(s));
    const int64_t refs = tail[0] + tail[1];
    if (refs < nt || refs > (int64_t)INT32_MAX / 4) return RQ_ERR_INVALID_ARG;
    if (refs > nt) {
        rm.arena.add(&rm.v, refs * 6);
        rm.arena.add(&rm.idx, refs * 3);
        rm.arena.add(&rm.tri, refs);
        RQ_CUDA(rm.arena.make(pool, s));
        split_kernel<<<blocks_of(nt, 128), 128, 0, s>>>(v, idx, nt, sb, pieces, off, rm.v, rm.idx, rm.tri);
        RQ_CUDA(cudaGetLastError());
        rm.n = refs;
    }
    return RQ_OK;
}

static rq_status build_scene(const float* vertices, int64_t nv, const int32_t* indices, int64_t nt, int method,
                             int optimize_passes, int split_budget, rq_scene_t* out, cudaMemPool_t pool, int device,
                             cudaStream_t s);

extern "C" rq_status rq_build_scene_gpu(const float* vertices, int64_t nv, const int32_t* indices, int64_t nt,
                                        int method, int optimize_passes, int split_budget, rq_scene_t* out,
                                        void* stream) {
    if (!out || !vertices || !indices || nv <= 0 || nt <= 0 || nt > (int64_t)INT32_MAX / 4) return RQ_ERR_INVALID_ARG;
    const bool thread_treelets = (method & RQ_GPU_BUILD_THREAD_TREELETS) != 0;
    method &= ~RQ_GPU_BUILD_THREAD_TREELETS;
    if (method != RQ_GPU_BUILD_LBVH && method != RQ_GPU_BUILD_PLOC) return RQ_ERR_INVALID_ARG;
    if (split_budget < 0 || split_budget > 400) return RQ_ERR_INVALID_ARG;
    int device = 0;
    RQ_CUDA(cudaGetDevice(&device));
    cudaMemPool_t pool = nullptr;
    {
        const cudaError_t e = scratch_pool().enter(device, &pool);
        if (e != cudaSuccess) return cuda_fail(e, "rq_build_scene_gpu: scratch pool");
    }
    const rq_status st = build_scene(vertices, nv, indices, nt, method | (thread_treelets ? RQ_GPU_BUILD_THREAD_TREELETS : 0),
                                     optimize_passes, split_budget, out, pool, device, (cudaStream_t)stream);
    if (st != RQ_OK) {  // otherwise the scene leaves, when it is destroyed
        cudaStreamSynchronize((cudaStream_t)stream);  // the frees queued on it are done
        scratch_pool().leave(device);
    }
    return st;
}

static rq_status build_scene(const float* vertices, int64_t nv, const int32_t* indices, int64_t nt, int method,
                             int optimize_passes, int split_budget, rq_scene_t* out, cudaMemPool_t pool, int device,
                             cudaStream_t s) {
    const bool thread_treelets = (method & RQ_GPU_BUILD_THREAD_TREELETS) != 0;
    method &= ~RQ_GPU_BUILD_THREAD_TREELETS;
    {
        // indices first: every kernel below reads vertices through them
        unsigned* bad_d = nullptr;
        unsigned bad = 0;
        Arena arena;
        arena.add(&bad_d, 1);
        RQ_CUDA(arena.make(pool, s));
        RQ_CUDA(cudaMemsetAsync(bad_d, 0, sizeof(unsigned), s));
        check_indices_kernel<<<std::min<unsigned>(blocks_of(3 * nt, 256), 8 * 148), 256, 0, s>>>(indices, 3 * nt, nv,
                                                                                                 bad_d);
        RQ_CUDA(cudaGetLastError());
        RQ_CUDA(cudaMemcpyAsync(&bad, bad_d, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        RQ_CUDA(cudaStreamSynchronize(s));
        if (bad) return RQ_ERR_INVALID_ARG;
    }
    RefMesh rm;
    if (split_budget > 0) {
        const rq_status ps = presplit(vertices, indices, nt, split_budget, rm, pool, s);
        if (ps != RQ_OK) return ps;
    }
    // The tree stages read boxes from the box mesh when the triangles were
    // split, from the triangles otherwise; leaves map back through rm.tri.
    const float* bv = rm.n ? rm.v : vertices;
    const int32_t* bi = rm.n ? rm.idx : indices;
    const int64_t n = rm.n ? rm.n : nt;
    int idx_bits = 1;
    while ((1ll << idx_bits) < n) ++idx_bits;
    const uint64_t idx_mask = (1ull << idx_bits) - 1;
    const int axis_bits = std::min(21, (64 - idx_bits) / 3);
    const int end_bit = idx_bits + 3 * axis_bits;
    rq_status st = RQ_OK;
    auto ok = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess && st == RQ_OK) st = cuda_fail(e, what);
        return st == RQ_OK;
    };
    const int64_t node_cap = std::max<int64_t>(1, n);  // an 8-wide node per binary node at most
    constexpr size_t kPad = 256;
    // device scratch, one allocation
    uint64_t *keys = nullptr, *keys_sorted = nullptr;
    BNode* bn = nullptr;
    NodeBox* leaves = nullptr;
    int32_t *leaf_parent = nullptr, *arrivals = nullptr;
    CollapseDP* dp = nullptr;
    unsigned* ob = nullptr;
    Item* queue[2] = {nullptr, nullptr};
    Levels* lv = nullptr;
    char* cub_temp = nullptr;
    PlocBuffers ploc;
    size_t cub_bytes = 0;
    Arena arena;
    // The keys hold the triangle numbers in order below the Morton codes, so a
    // stable sort by the codes alone orders them.
    ok(cub::DeviceRadixSort::SortKeys(nullptr, cub_bytes, keys, keys_sorted, (int)n, idx_bits, end_bit, s),
       "rq_build_scene_gpu");
    arena.add(&keys, n);
    arena.add(&keys_sorted, n);
    arena.add(&bn, n - 1);
    arena.add(&leaves, n);
    arena.add(&leaf_parent, n);
    arena.add(&arrivals, n - 1);
    arena.add(&dp, n - 1);
    arena.add(&ob, 6);
    arena.add(&queue[0], node_cap);
    arena.add(&queue[1], node_cap);
    arena.add(&lv, 1);
    arena.add(&cub_temp, (int64_t)cub_bytes);
    if (method == RQ_GPU_BUILD_PLOC) ploc.layout(arena, n);
    // the scene's buffers, one allocation of its own
    char* block = nullptr;
    const size_t node_bytes = ((size_t)node_cap * 80 + kPad + 255) / 256 * 256;
    const size_t woop_bytes = ((size_t)n * 48 + kPad + 255) / 256 * 256;
    float4 *nodes = nullptr, *woop = nullptr;
    int32_t* prim = nullptr;
    if (st == RQ_OK && ok(arena.make(pool, s), "rq_build_scene_gpu") &&
        ok(cudaMalloc(&block, node_bytes + woop_bytes + (size_t)n * 12), "rq_build_scene_gpu")) {
        nodes = (float4*)block;
        woop = (float4*)(block + node_bytes);
        prim = (int32_t*)(block + node_bytes + woop_bytes);
        const unsigned init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
        ok(cudaMemcpyAsync(ob, init, sizeof(init), cudaMemcpyHostToDevice, s), "rq_build_scene_gpu");
        ok(cudaMemsetAsync(woop + 3 * n, 0, kPad, s), "rq_build_scene_gpu");
        ok(cudaMemsetAsync(prim, 0xFF, n * 12, s), "rq_build_scene_gpu");
        ok(cudaMemsetAsync(arrivals, 0, std::max<int64_t>(1, n - 1) * sizeof(int32_t), s), "rq_build_scene_gpu");
        ok(cudaMemsetAsync(lv, 0, sizeof(Levels), s), "rq_build_scene_gpu");
    }
    if (st == RQ_OK) {
        centroid_bounds_kernel<<<std::min<unsigned>(blocks_of(n, 256), 4 * 148), 256, 0, s>>>(bv, bi, n, ob);
        morton_kernel<<<blocks_of(n, 256), 256, 0, s>>>(bv, bi, n, ob, axis_bits, idx_bits, keys);
        ok(cudaGetLastError(), "rq_build_scene_gpu");
        ok(cub::DeviceRadixSort::SortKeys(cub_temp, cub_bytes, keys, keys_sorted, (int)n, idx_bits, end_bit, s),
           "rq_build_scene_gpu");
        leaf_boxes_kernel<<<blocks_of(n, 256), 256, 0, s>>>(keys_sorted, idx_mask, n, bv, bi, leaves);
        ok(cudaGetLastError(), "rq_build_scene_gpu");
    }
    int64_t n_nodes = 1;
    if (st == RQ_OK && n > 1) {
        if (method == RQ_GPU_BUILD_PLOC) {
            st = ploc_tree(ploc, n, leaves, bn, leaf_parent, s);
        } else {
            radix_tree_kernel<<<blocks_of(n - 1, 256), 256, 0, s>>>(keys_sorted, n, bn, leaf_parent);
            boxes_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, leaves, bn, leaf_parent, arrivals);
            ok(cudaGetLastError(), "rq_build_scene_gpu");
        }
        for (int pass = 0; pass < optimize_passes && st == RQ_OK; ++pass) {
            ok(cudaMemsetAsync(arrivals, 0, (n - 1) * sizeof(int32_t), s), "rq_build_scene_gpu");
            if (thread_treelets)
                treelet_kernel<<<blocks_of(n, 128), 128, 0, s>>>(n, leaves, bn, leaf_parent, arrivals, kTreeletLeaves);
            else
                treelet_warp_kernel<<<blocks_of(n, kTreeletWarpBlock), kTreeletWarpBlock, 0, s>>>(
                    n, leaves, bn, leaf_parent, arrivals, kTreeletLeaves,
                    pass < 65535 ? (unsigned)pass + 1u : 1u);  // pass 1 takes every treelet; stamps have 16 bits
            ok(cudaGetLastError(), "rq_build_scene_gpu");
        }
        if (st == RQ_OK) {
            ok(cudaMemsetAsync(arrivals, 0, (n - 1) * sizeof(int32_t), s), "rq_build_scene_gpu");
            collapse_dp_kernel<<<blocks_of(n, 256), 256, 0, s>>>(n, leaves, bn, leaf_parent, arrivals, dp);
            ok(cudaGetLastError(), "rq_build_scene_gpu");
        }
    }
    if (st == RQ_OK) {
        // level 0: the root (binary node 0, or the single triangle)
        const Item root{n > 1 ? 0 : ~0, 0};
        const unsigned long long one = 1ull;
        ok(cudaMemcpyAsync(queue[0], &root, sizeof(root), cudaMemcpyHostToDevice, s), "rq_build_scene_gpu");
        ok(cudaMemcpyAsync(&lv->alloc[0], &one, sizeof(one), cudaMemcpyHostToDevice, s), "rq_build_scene_gpu");
        // An 8-wide tree of n triangles: eight levels ahead are rarely too many.
        constexpr int kAhead = 8;
        const unsigned grid = std::min<unsigned>(blocks_of(node_cap, kExpandBlock / 8), 148 * 8);
        unsigned error = 0u;
        unsigned long long left = 1ull;
        for (int level = 0; st == RQ_OK && left != 0;) {
            if (level + kAhead > kMaxLevels) {
                st = RQ_ERR_BAD_SCENE;
                break;
            }
            for (int q = 0; q < kAhead; ++q, ++level)
                expand_kernel<<<grid, kExpandBlock, 0, s>>>(level, queue[level & 1], queue[(level + 1) & 1], bn, leaves,
                                                            keys_sorted, idx_mask, rm.tri, nodes, (unsigned)node_cap, prim,
                                                            (unsigned)n, lv, n > 1 ? dp : nullptr);
            unsigned total = 0u;
            ok(cudaGetLastError(), "rq_build_scene_gpu");
            ok(cudaMemcpyAsync(&left, &lv->alloc[level], sizeof(left), cudaMemcpyDeviceToHost, s), "rq_build_scene_gpu");
            ok(cudaMemcpyAsync(&total, &lv->node_base[level], sizeof(total), cudaMemcpyDeviceToHost, s),
               "rq_build_scene_gpu");
            ok(cudaMemcpyAsync(&error, &lv->error, sizeof(error), cudaMemcpyDeviceToHost, s), "rq_build_scene_gpu");
            ok(cudaStreamSynchronize(s), "rq_build_scene_gpu");
            left &= 0xFFFFFFFFull;
            n_nodes = (int64_t)total + (int64_t)left;
            if (st == RQ_OK && error) st = RQ_ERR_BAD_SCENE;  // capacity exceeded: cannot happen for a valid tree
        }
        if (st == RQ_OK) {
            woop_rows_kernel<<<blocks_of(n, 128), 128, 0, s>>>(n, vertices, indices, woop, prim);
            ok(cudaGetLastError(), "rq_build_scene_gpu");
            ok(cudaMemsetAsync(nodes + 5 * n_nodes, 0, kPad, s), "rq_build_scene_gpu");
        }
    }
    float root[20] = {};
    if (st == RQ_OK)
        ok(cudaMemcpyAsync(root, nodes, sizeof(root), cudaMemcpyDeviceToHost, s), "rq_build_scene_gpu");
    ok(cudaStreamSynchronize(s), "rq_build_scene_gpu");
    // The pool gives back only what the host has seen the stream let go of, so
    // the scene keeps an event behind the frees and waits for it when it goes.
    // (Freeing before the wait above instead has the pool give back all beyond
    // kPoolKeepBytes in every build and map it again in the next: 2M triangles
    // 9.9 -> 11.5 ms.)
    cudaEvent_t freed = nullptr;
    if (st == RQ_OK) ok(cudaEventCreateWithFlags(&freed, cudaEventDisableTiming), "rq_build_scene_gpu");
    arena.release();
    rm.arena.release();
    if (st == RQ_OK) ok(cudaEventRecord(freed, s), "rq_build_scene_gpu");
    if (st != RQ_OK) {
        if (freed) cudaEventDestroy(freed);
        cudaFree(block);
        return st;
    }
    rq_scene* sc = new rq_scene();
    sc->kind = RQ_BVH_CWBVH;
    sc->device = device;
    sc->block = block;
    sc->scratch_freed = freed;
    sc->nodes = nodes;
    sc->woop = woop;
    sc->prim_index = prim;
    sc->node_f4 = n_nodes * 5;
    sc->woop_f4 = n * 3;
    sc->prim_count = n * 3;
    sc->owned = true;
    uint32_t ew;
    std::memcpy(&ew, &root[3], 4);
    for (int a = 0; a < 3; ++a) {
        const int e = (int)(int8_t)((ew >> (8 * a)) & 0xFFu);
        sc->lo[a] = root[a];
        sc->hi[a] = root[a] + 255.0f * std::ldexp(1.0f, e);
    }
    *out = sc;
    return RQ_OK;
}
