// Persistent trace kernels for sm_100a: the compressed 8-wide BVH (CWBVH) and
// the binary BVH (BVH2), closest-hit and any-hit, over one scene or over a
// batch of (scene, rays) items in one launch.
//
// Work distribution (both kernels).  One CTA per SM slot stays resident for the
// whole launch.  A warp hands rays to its idle lanes from one 64-bit global
// counter: the lanes that need a ray vote, one lane adds their count to the
// counter and broadcasts the old value (the reference's per-warp atomicAdd,
// src/TraversalKernelCWBVH.cu:56-87, written with __shfl_sync instead of a
// volatile shared word so it is correct under independent thread scheduling).
// A warp re-fills after the idle lanes have cost Nw lane-iterations beyond Nd
// (src/TraversalKernelCWBVH.cu:365-371).  Large CWBVH any-hit batches take
// their rays through a per-warp ring of prefetched rays instead (below), and
// the last rays of a CWBVH launch get four lanes each.  Every vote is over the
// full warp and every loop is warp-uniform, so lanes never diverge around a
// collective.
//
// Safety.  A ray whose stack would overflow, whose node/triangle index falls
// outside the buffers, or that runs more than the step limit is finished as
// a miss and the context's error word records why; the kernel itself never
// reads outside the buffers it was given and never spins without a bound.
#include <cstdio>

#include "device_api.h"
#include "trace_common.cuh"

namespace rq {

constexpr int kStackTotal = 64;  // entries per lane (shared + local)
constexpr int kDeeperMinLanes = 16;  // any-hit: lanes that make a second node step worth its issue slots

// The persistent CWBVH kernel's last rays: once the counter is used up and at
// most 8 of a warp's rays are left, four lanes take each (lanes_loop).
constexpr int kTailLanes = 4, kTailRays = 32 / kTailLanes;

#ifdef RQ_MAXNREG
#define RQ_CW_BOUNDS __maxnreg__(RQ_MAXNREG)  // register cap (occupancy experiments)
#define RQ_BVH2_BOUNDS __maxnreg__(RQ_MAXNREG)
#else
#define RQ_CW_BOUNDS __maxnreg__(COUNT ? 64 : 56)  // see park_bytes_per_warp
// The BVH2 kernel fits 56 registers without spilling (nine 128-thread blocks
// per SM instead of eight): closest-hit +2.3 %, any-hit unchanged on the
// small scene; 48 spills and loses 2 % any-hit.
#define RQ_BVH2_BOUNDS __maxnreg__(56)
#endif
constexpr uint32_t kBvh2Sentinel = 0x76543210u;  // src/TraversalKernelBVH2.cu:33

// ------------------------------------------------- per-warp ray prefetch --
//
// The CWBVH any-hit kernel of large batches (RING) takes rays 32 at a time per
// warp (one counter add per 32 rays) into a ring of 64 slots per warp in
// shared memory: two halves, each filled by one cp.async group (every lane
// copies one ray's 32 bytes and notes its batch item).  A refill hands idle
// lanes the next slots in order; the ray loads of a half were issued a refill
// or more earlier and no longer stall the warp, and neither a counter add nor
// the item search sits on its path.  A half is refilled as soon as its last
// slot is handed out.  The last rays of a launch stay tied to the warp whose
// ring holds them, which costs a short launch more than the ring saves, so it
// is used from kRingMinRaysPerThread rays per thread of the grid up.  12 scenes,
// us without / with the ring: 1.2M rays (7 per thread) 222 / 239, 2.3M (14) 379
// / 389, 3.9M (23) 645 / 640, 7.9M (46) 1,183 / 1,155.  One scene has no item
// search to save and loses 1 % even at 64M rays (17,644 / 17,861 on 4M
// triangles, 11,715 / 11,795 on 100,000).  Any-hit only: closest-hit batches
// measured 1 % slower with the ring.
constexpr unsigned kRingHalf = 32;  // rays per counter add
constexpr unsigned kRingSlots = 2 * kRingHalf;
// rays [64][2] float4, the two halves' first global ray index, items [64]
constexpr size_t kRingBytesPerWarp = kRingSlots * sizeof(Ray) + 2 * sizeof(int64_t) + kRingSlots * sizeof(int);
static_assert(kRingBytesPerWarp % 16 == 0, "ring keeps 16 B alignment");

// A CWBVH ray's values that only its end or a rare branch reads wait in shared
// memory, a word per lane each: hit address, u, v, result index (two words),
// and for a batch its item, the prefetched item and the item's Woop limit.  With
// them in registers the kernels took 64 and eight 128-thread blocks fit an SM;
// without, 56 and nine, with no spills (10 B in the ring batch kernel with more
// than four stack entries; 72 registers and seven blocks are 1-6 % slower than
// 64, 48 and ten spill and are 2-10 % slower).  Single-scene kernels read the
// limits from the launch parameters.  4.2M city primary rays 808 -> 795 us, 4M AO rays on 4M triangles
// 1,240 -> 1,204 us, 1M closest hits 390 -> 389 us, 18M AO rays of 12 scenes
// 3,332 -> 3,205 us (with four stack entries, see launch_trace).
constexpr int kParkWordsSingle = 5, kParkWordsMulti = 8;
__host__ __device__ constexpr size_t park_bytes_per_warp(bool multi) {
    return (multi ? kParkWordsMulti : kParkWordsSingle) * 32 * sizeof(int);
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The batch item holding global ray g, searching forward from `hint` (the
// item of a smaller ray index taken by the same lane; -1 for none).
__device__ __forceinline__ int find_item(const TraceParams& p, int64_t g, int hint) {
    int lo = hint, hi = p.n_items - 1;
    if (lo < 0 || lo > hi || p.items[lo].ray_begin > g) lo = 0;
    if (lo < hi && p.items[lo + 1].ray_begin <= g) {
        ++lo;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (p.items[mid].ray_begin <= g) lo = mid; else hi = mid - 1;
        }
    }
    return lo;
}

// Resolves a global ray index to its item (batch) and loads the ray.
struct Lane {
    const float4* nodes;
    const float4* woop;
    int64_t out_idx;
    int64_t gidx;
    int item;  // batch item of the ray (its hit buffer or AO counters are read at the end)
    uint32_t node_limit, woop_limit;
};

// Points a lane at global ray g of batch item `item` (0 for a single scene)
// and returns the item.
template <bool MULTI>
__device__ __forceinline__ const TraceItem* set_lane(const TraceParams& p, int64_t g, int item, Lane& L) {
    const TraceItem* it = MULTI ? p.items + item : &p.single;
    const int64_t local = g - (MULTI ? it->ray_begin : 0);
    L.item = item;
    L.nodes = it->nodes;
    L.woop = it->woop;
    L.node_limit = it->node_limit;
    L.woop_limit = it->woop_limit;
    L.out_idx = it->perm ? (int64_t)__ldg(it->perm + local) : local;
    L.gidx = g;
    return it;
}

template <bool MULTI>
__device__ __forceinline__ Ray fetch_ray(const TraceParams& p, int64_t g, Lane& L) {
    // A lane's rays come from a counter that only grows, so its next ray is in
    // its current item or a later one: check the next item's start first, and
    // search only forward when the ray lies beyond it.
    const TraceItem* it = set_lane<MULTI>(p, g, MULTI ? find_item(p, g, L.item) : 0, L);
    const int64_t local = g - (MULTI ? it->ray_begin : 0);
    Ray r;
    r.origin_tmin = __ldcs(&it->rays[local].origin_tmin);
    r.dir_tmax = __ldcs(&it->rays[local].dir_tmax);
    return r;
}

__device__ __forceinline__ void store_hit(Hit* hits, int64_t i, float t, int addr, float u, float v) {
    __stcs(&hits[i].t_triId_u_v, make_float4(t, __int_as_float(addr), u, v));
}

// A finished ray's result: its Hit, or -- for an item with AO counters -- one
// count for its surfel when it is occluded.
template <bool MULTI>
__device__ __forceinline__ void finish_ray(const TraceParams& p, int item, int64_t out_idx, float t, int addr, float u,
                                           float v) {
    const TraceItem* it = MULTI ? p.items + item : &p.single;
    uint32_t* counts = it->ao_counts;
    if (counts) {
        if (addr >= 0) atomicAdd(counts + out_idx / it->ao_spp, 1u);
    } else {
        store_hit(it->hits, out_idx, t, addr, u, v);
    }
}
template <bool MULTI>
__device__ __forceinline__ void finish_ray(const TraceParams& p, const Lane& L, float t, int addr, float u, float v) {
    finish_ray<MULTI>(p, L.item, L.out_idx, t, addr, u, v);
}

// ------------------------------------ CWBVH, several lanes to a ray --
//
// Where the warps don't fill the GPU, a launch is bound by the latency of the
// longest ray, and in cwbvh_kernel a lane works through a node's eight children
// (and then its triangles) one after the other: about 2,000 cycles per node with
// one warp per scheduler.  Here G = 8 or 4 lanes share a ray: lane c tests the
// children whose hit bits are 24 + c * 8 / G and up and those of their
// triangles it hits, and the lanes vote.  The ray, the node group and the stack
// pointer are replicated over the lanes.
//
// The order is the oracle's: nearest child first, all triangles of a node
// before its children, and of a group's triangles the closest hit (any-hit:
// the first hit) in the group's order, so hits are bit-identical to
// rq_trace_ordered's.  Every lane of a group takes the same decisions about
// its ray; the loop itself is warp-uniform.
//
// push(ng), pop(): the group's stack, shared entries written by lane 0.
// hit(t, addr, u, v): a closest-hit ray's new best (which sets tmax), the end
// of an any-hit ray.  done(err): the end of a ray without one.
template <bool ANY, int G, bool TAIL, class Limit, class Push, class Pop, class Hit_, class Done>
__device__ __forceinline__ void lanes_loop(const float4* nodes, const float4* woop, uint32_t node_limit,
                                           int step_limit, float ox, float oy, float oz, float dx, float dy,
                                           float dz, float idx_, float idy, float idz, unsigned octinv, float tmin,
                                           float& tmax, uint2& ng, int& sp, int& steps, bool& active,
                                           const Limit& woop_limit, const Push& push, const Pop& pop, const Hit_& hit,
                                           const Done& done) {
    constexpr int C = 8 / G;  // children per lane
    const unsigned lane = threadIdx.x & 31u;
    const unsigned c = lane % G, group_shift = lane - c;
    const bool negx = idx_ < 0.f, negy = idy < 0.f, negz = idz < 0.f;
    while (__any_sync(kFullMask, active)) {
        unsigned fault = 0u, leaf_bits = 0u, inner = 0u;
        uint2 next = make_uint2(0u, 0u);  // child base, imask
        uint32_t tri_base = 0u;
        if (active && (!TAIL || ng.y > 0x00FFFFFFu)) {
            const unsigned hitsm = ng.y;
            const unsigned bit = highest_bit(hitsm);
            const unsigned base = ng.x;
            ng.y &= ~(1u << bit);
            if (ng.y > 0x00FFFFFFu && !push(ng)) fault = kErrStackOverflow;
            const unsigned slot = (bit - 24u) ^ octinv;
            const unsigned ci = base + (unsigned)__popc(hitsm & ~(0xFFFFFFFFu << slot));
            if (++steps > step_limit) fault |= kErrTimeout;
            if (ci >= node_limit) fault |= kErrBadScene;
            if (!fault) {
                const float4* np = nodes + (size_t)ci * 5u;
                const float4 n0 = ld_nc(np + 0), n1 = ld_nc(np + 1), n2 = ld_nc(np + 2);
                const float4 n3 = ld_nc(np + 3), n4 = ld_nc(np + 4);
                const unsigned ew = __float_as_uint(n0.w);
                const float adjx = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)(ew & 0xFFu) + 127)) << 23), idx_);
                const float adjy = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)((ew >> 8) & 0xFFu) + 127)) << 23), idy);
                const float adjz = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)((ew >> 16) & 0xFFu) + 127)) << 23), idz);
                const float orx = __fmul_rn(-__fsub_rn(ox, n0.x), idx_);
                const float ory = __fmul_rn(-__fsub_rn(oy, n0.y), idy);
                const float orz = __fmul_rn(-__fsub_rn(oz, n0.z), idz);
#pragma unroll
                for (int q = 0; q < C; ++q) {
                    const unsigned pos = c * C + q;         // hit bit 24 + pos
                    const unsigned child = pos ^ octinv;    // its slot
                    auto child_byte = [&](float w0, float w1) -> unsigned {
                        return __byte_perm(__float_as_uint(w0), __float_as_uint(w1), child) & 0xFFu;
                    };
                    const unsigned meta = child_byte(n1.z, n1.w);
                    const float qlx = __uint2float_rn(child_byte(n2.x, n2.y)), qhx = __uint2float_rn(child_byte(n3.z, n3.w));
                    const float qly = __uint2float_rn(child_byte(n2.z, n2.w)), qhy = __uint2float_rn(child_byte(n4.x, n4.y));
                    const float qlz = __uint2float_rn(child_byte(n3.x, n3.y)), qhz = __uint2float_rn(child_byte(n4.z, n4.w));
                    const float tx0 = __fmaf_rn(negx ? qhx : qlx, adjx, orx), tx1 = __fmaf_rn(negx ? qlx : qhx, adjx, orx);
                    const float ty0 = __fmaf_rn(negy ? qhy : qly, adjy, ory), ty1 = __fmaf_rn(negy ? qly : qhy, adjy, ory);
                    const float tz0 = __fmaf_rn(negz ? qhz : qlz, adjz, orz), tz1 = __fmaf_rn(negz ? qlz : qhz, adjz, orz);
                    const float cmin = fmaxf(imax3(tx0, ty0, tz0), tmin);
                    const float cmax = fminf(imin3(tx1, ty1, tz1), tmax);
                    if (cmin <= cmax) {
                        // meta: 0x20 | (24 + slot) for an inner child, unary count << 5 | offset for a leaf
                        if ((meta & 0x18u) == 0x18u) inner |= (meta >> 5 ? 1u : 0u) << pos;
                        else leaf_bits |= (meta >> 5) << (meta & 0x1Fu);
                    }
                }
                next = make_uint2(__float_as_uint(n1.x), ew >> 24);
                tri_base = __float_as_uint(n1.y);
            }
        } else if (TAIL && active) {  // a postponed triangle group: every G-th triangle
            tri_base = ng.x;
            for (unsigned k = G - c, b = ng.y; b; ++k) {
                const unsigned top = 1u << highest_bit(b);
                if (k % G == 0u) leaf_bits |= top;
                b &= ~top;
            }
        }
        unsigned inner_hits = inner;
        if (G == 8) {
            inner_hits = (__ballot_sync(kFullMask, inner != 0u) >> group_shift) & 0xFFu;
        } else {
#pragma unroll
            for (int m = G / 2; m > 0; m >>= 1) inner_hits |= __shfl_xor_sync(kFullMask, inner_hits, m);
        }

        if (active) {
            if (fault) {
                leaf_bits = 0u;
                done(fault);
            } else {
                ng = make_uint2(next.x, (inner_hits << 24) | next.y);
            }
        }

        // Triangles of this lane, highest bit first.
        if (__any_sync(kFullMask, leaf_bits != 0u)) {
            float bt = tmax, bu = 0.f, bv = 0.f;
            int order = -1, addr = -1;  // group position and address of the lane's best hit
            bool bad = false;
            while (leaf_bits) {
                const unsigned ti = highest_bit(leaf_bits);
                leaf_bits &= ~(1u << ti);
                const unsigned tri = tri_base * 3u + ti * 3u;
                if (tri >= woop_limit()) {
                    bad = true;
                    order = (int)ti;
                    break;
                }
                const float4* tp = woop + tri;
                const float4 v0 = ld_nc(tp), v1 = ld_nc(tp + 1), v2 = ld_nc(tp + 2);
                float t, u, v;
                if (woop_test(v0, v1, v2, ox, oy, oz, dx, dy, dz, tmin, bt, t, u, v)) {
                    bt = t;
                    bu = u;
                    bv = v;
                    addr = (int)tri;
                    order = (int)ti;
                    if (ANY) break;
                }
            }
            __syncwarp();
            if (__any_sync(kFullMask, order >= 0)) {
                // The winner of the group: any-hit the first in order, closest
                // the smallest t, the first in order among equals.  A triangle
                // outside the buffer ends the ray where its turn comes.
                float wt = order >= 0 ? bt : 0.f;
                int wo = order;
                bool wbad = bad;
#pragma unroll
                for (int m = G / 2; m > 0; m >>= 1) {
                    const float t2 = __shfl_xor_sync(kFullMask, wt, m);
                    const int o2 = __shfl_xor_sync(kFullMask, wo, m);
                    const bool b2 = __shfl_xor_sync(kFullMask, (int)wbad, m) != 0;
                    bool take;
                    if (ANY) take = o2 > wo;
                    else take = o2 >= 0 && (wo < 0 || (b2 != wbad ? b2 : (t2 < wt || (t2 == wt && o2 > wo))));
                    if (take) {
                        wt = t2;
                        wo = o2;
                        wbad = b2;
                    }
                }
                const unsigned won = __ballot_sync(kFullMask, order >= 0 && order == wo && bad == wbad);
                const unsigned mine = (won >> group_shift) & ((1u << G) - 1u);
                const int src = mine ? (int)group_shift + __ffs(mine) - 1 : (int)lane;
                const float u2 = __shfl_sync(kFullMask, bu, src), v2 = __shfl_sync(kFullMask, bv, src);
                const int a2 = __shfl_sync(kFullMask, addr, src);
                if (active && wo >= 0) {
                    if (wbad) done(kErrBadScene);
                    else hit(wt, a2, u2, v2);
                }
            }
        }

        __syncwarp();  // the group's pushes are visible to its lanes
        if (active && ng.y <= 0x00FFFFFFu) {
            if (sp > 0) ng = pop();
            else done(0u);
        }
        __syncwarp();  // and read before a lane pushes over them
    }
}

// ------------------------------------------------------------------ CWBVH --

template <bool ANY, int SMEM, bool MULTI, bool COUNT, bool RING>
__global__ void RQ_CW_BOUNDS cwbvh_kernel(const TraceParams p) {
    extern __shared__ uint2 sstack[];
    constexpr int LOCAL = kStackTotal - SMEM;
    uint2 lstack[LOCAL];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned tid = threadIdx.x;
    const unsigned B = blockDim.x;

    static_assert(MULTI || !RING, "the ring is for batches");
    Lane L{};
    float ox = 0.f, oy = 0.f, oz = 0.f, dx = 0.f, dy = 0.f, dz = 0.f, tmin = 0.f, tmax = 0.f;
    float idx_ = 0.f, idy = 0.f, idz = 0.f;
    unsigned octinv = 0;
    uint2 ng = make_uint2(0u, 0u), tg = make_uint2(0u, 0u);
    int sp = 0, steps = 0, nvis = 0, ntri = 0;
    bool active = false, exhausted = false;
    const float rt = p.postpone_ratio;

    auto push = [&](uint2 v) -> bool {
        if (sp < SMEM) sstack[(unsigned)sp * B + tid] = v;
        else if (sp < kStackTotal) lstack[sp - SMEM] = v;
        else return false;
        ++sp;
        return true;
    };
    auto pop = [&]() -> uint2 {
        --sp;
        return sp < SMEM ? sstack[(unsigned)sp * B + tid] : lstack[sp - SMEM];
    };
    // What only the end of a ray reads waits in shared memory, not in registers.
    int* parked = reinterpret_cast<int*>(sstack + (size_t)SMEM * B) +
                  (tid >> 5) * (unsigned)(park_bytes_per_warp(MULTI) / sizeof(int)) + lane;
    auto woop_limit = [&]() -> unsigned { return MULTI ? (unsigned)parked[224] : p.single.woop_limit; };
    auto park_hit = [&](int addr, float u, float v) {
        parked[0] = addr;
        parked[32] = __float_as_int(u);
        parked[64] = __float_as_int(v);
    };
    auto end_ray = [&](float t, int addr, float u, float v) {
        const int64_t out = (int64_t)(((uint64_t)(unsigned)parked[128] << 32) | (unsigned)parked[96]);
        finish_ray<MULTI>(p, MULTI ? parked[160] : 0, out, t, addr, u, v);
        if (COUNT) {
            p.node_visits[L.gidx] = nvis;
            p.tri_tests[L.gidx] = ntri;
        }
        active = false;
    };
    auto finish = [&](unsigned err) {
        if (err) atomicOr(&p.scratch->error, err);
        if (ANY) end_ray(tmax, -1, 0.f, 0.f);
        else end_ray(tmax, err ? -1 : parked[0], __int_as_float(parked[32]), __int_as_float(parked[64]));
    };

    // Per-warp ray ring after the stacks.
    unsigned char* const ring = reinterpret_cast<unsigned char*>(sstack + (size_t)SMEM * B) +
                                (size_t)(B >> 5) * park_bytes_per_warp(MULTI) + (size_t)(tid >> 5) * kRingBytesPerWarp;
    float4* const ring_ray = reinterpret_cast<float4*>(ring);
    int64_t* const ring_base = reinterpret_cast<int64_t*>(ring + kRingSlots * sizeof(Ray));
    int* const ring_item = reinterpret_cast<int*>(ring + kRingSlots * sizeof(Ray) + 2 * sizeof(int64_t));
    unsigned cons = 0u;  // next slot to hand out (warp-uniform)
    // parked[192]: item of the lane's last prefetched ray (forward search hint)
    if (RING) parked[192] = -1;
    // Takes the next 32 rays from the counter into half `half` of the ring.
    auto claim = [&](unsigned half) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&p.scratch->ray_counter, (unsigned long long)kRingHalf);
        base = __shfl_sync(kFullMask, base, 0);
        if (lane == 0) ring_base[half] = (int64_t)base;
        const int64_t g = (int64_t)base + lane;
        if (g < p.total_rays) {
            const unsigned slot = half * kRingHalf + lane;
            const int item = find_item(p, g, parked[192]);
            parked[192] = item;
            ring_item[slot] = item;
            const TraceItem* it = p.items + item;
            const Ray* src = it->rays + (g - it->ray_begin);
            cp_async16(ring_ray + 2u * slot, &src->origin_tmin);
            cp_async16(ring_ray + 2u * slot + 1u, &src->dir_tmax);
        }
        cp_async_commit();
    };
    if (RING) {
        claim(0u);
        claim(1u);
    }
    auto start = [&](const Ray& r) {
        ox = r.origin_tmin.x; oy = r.origin_tmin.y; oz = r.origin_tmin.z; tmin = r.origin_tmin.w;
        dx = r.dir_tmax.x; dy = r.dir_tmax.y; dz = r.dir_tmax.z; tmax = r.dir_tmax.w;
        idx_ = guarded_rcp(dx);
        idy = guarded_rcp(dy);
        idz = guarded_rcp(dz);
        octinv = 7u - (((dx < 0.f) ? 4u : 0u) | ((dy < 0.f) ? 2u : 0u) | ((dz < 0.f) ? 1u : 0u));
        ng = make_uint2(0u, 0x80000000u);
        tg = make_uint2(0u, 0u);
        sp = 0; steps = 0; nvis = 0; ntri = 0;
        if (!ANY) park_hit(-1, 0.f, 0.f);
        parked[96] = (int)(unsigned)L.out_idx;
        parked[128] = (int)(unsigned)((uint64_t)L.out_idx >> 32);
        if (MULTI) {
            parked[160] = L.item;
            parked[224] = (int)p.items[L.item].woop_limit;
        }
        active = true;
    };

    for (;;) {
        // ---- hand rays to idle lanes
        const bool need = !active && !exhausted;
        const unsigned needm = __ballot_sync(kFullMask, need);
        if (RING && needm) {
            // Slots [cons, end) go to the needy lanes in lane order.  The half
            // holding cons was filled before the other one, so its copies are
            // done after waiting for all but the newest group; a refill that
            // runs into the other half waits for that one too.
            const unsigned half_end = (cons & kRingHalf) + kRingHalf;
            const unsigned end = cons + (unsigned)__popc(needm);
            if (end > half_end) cp_async_wait<0>(); else cp_async_wait<1>();
            __syncwarp();
            if (need) {
                const unsigned rank = (unsigned)__popc(needm & lanemask_lt());
                const unsigned slot = (cons + rank) & (kRingSlots - 1u);
                const int64_t g = ring_base[slot / kRingHalf] + (slot & (kRingHalf - 1u));
                if (g < p.total_rays) {
                    set_lane<MULTI>(p, g, ring_item[slot], L);
                    Ray r;
                    r.origin_tmin = ring_ray[2u * slot];
                    r.dir_tmax = ring_ray[2u * slot + 1u];
                    start(r);
                } else {
                    exhausted = true;
                }
            }
            if (end >= half_end) {  // the half of cons is used up: refill it
                __syncwarp();
                claim((cons / kRingHalf) & 1u);
            }
            cons = end & (kRingSlots - 1u);
        } else if (needm) {
            const int leader = __ffs(needm) - 1;
            unsigned long long base = 0;
            if ((int)lane == leader) base = atomicAdd(&p.scratch->ray_counter, (unsigned long long)__popc(needm));
            base = __shfl_sync(kFullMask, base, leader);
            if (need) {
                const int64_t g = (int64_t)base + __popc(needm & lanemask_lt());
                if (g < p.total_rays) {
                    start(fetch_ray<MULTI>(p, g, L));
                } else {
                    exhausted = true;
                }
            }
        }
        const unsigned live = __ballot_sync(kFullMask, active);
        if (live == 0u) break;

        // ---- the launch's last rays: no more to fetch, few left in the warp.
        // A launch ends with warps that each carry a few long rays, a lane per
        // ray and the rest idle: about 55 us per launch.  Groups of lanes take
        // the rays over here, with the shared part of their stacks and what
        // they parked in place (a ray that has spilled past it to its lane's
        // local memory keeps the warp in the loop below until it has popped
        // that far).  us before / after: AO 94k, 262k, 524k rays on 200,000
        // triangles 74 / 67, 117 / 104, 165 / 149, closest-hit 149 / 136, 222 /
        // 201, 341 / 315; 1M AO rays on 10,592 215 / 204, 1M closest-hit on
        // 20,000 388 / 372, 4M AO rays on 4M 1,202 / 1,178, batches of 1.2M
        // and 7.9M rays 220 / 208, 1,151 / 1,145.  Eight lanes from 4 rays on
        // gain 60-75 % of that, two from 16 on 50-75 %.
        if (!COUNT && __any_sync(kFullMask, exhausted) && __popc(live) <= kTailRays &&
            !__any_sync(kFullMask, active && sp > SMEM)) {
            const unsigned c = lane % kTailLanes, group = lane / kTailLanes;
            unsigned m = live;
            for (unsigned k = group; m && k; --k) m &= m - 1u;
            const int src = m ? __ffs(m) - 1 : (int)lane;
            ox = __shfl_sync(kFullMask, ox, src);
            oy = __shfl_sync(kFullMask, oy, src);
            oz = __shfl_sync(kFullMask, oz, src);
            dx = __shfl_sync(kFullMask, dx, src);
            dy = __shfl_sync(kFullMask, dy, src);
            dz = __shfl_sync(kFullMask, dz, src);
            tmin = __shfl_sync(kFullMask, tmin, src);
            tmax = __shfl_sync(kFullMask, tmax, src);
            idx_ = __shfl_sync(kFullMask, idx_, src);
            idy = __shfl_sync(kFullMask, idy, src);
            idz = __shfl_sync(kFullMask, idz, src);
            octinv = __shfl_sync(kFullMask, octinv, src);
            ng.x = __shfl_sync(kFullMask, ng.x, src);
            ng.y = __shfl_sync(kFullMask, ng.y, src);
            sp = __shfl_sync(kFullMask, sp, src);
            steps = __shfl_sync(kFullMask, steps, src);
            active = m != 0u;
            parked += src - (int)lane;
            uint2* const column = sstack + (tid - lane + (unsigned)src);
            __syncwarp();  // what the rays' first lanes parked is visible
            const TraceItem* it = MULTI ? p.items + (m ? parked[160] : 0) : &p.single;
            lanes_loop<ANY, kTailLanes, true>(
                it->nodes, it->woop, it->node_limit, p.step_limit, ox, oy, oz, dx, dy, dz, idx_, idy,
                idz, octinv, tmin, tmax, ng, sp, steps, active, woop_limit,
                [&](uint2 v) {
                    if (sp < SMEM) {
                        if (c == 0u) column[(unsigned)sp * B] = v;
                    } else if (sp < kStackTotal) {
                        lstack[sp - SMEM] = v;
                    } else {
                        return false;
                    }
                    ++sp;
                    return true;
                },
                [&]() {
                    --sp;
                    return sp < SMEM ? column[(unsigned)sp * B] : lstack[sp - SMEM];
                },
                [&](float t, int addr, float u, float v) {
                    if (ANY) {
                        if (c == 0u) end_ray(t, addr, u, v);
                        active = false;
                    } else {
                        tmax = t;
                        if (c == 0u) park_hit(addr, u, v);
                    }
                },
                [&](unsigned err) {
                    if (c == 0u) finish(err);
                    active = false;
                });
            break;
        }

        int lost = 0;
        for (;;) {
            // ---- node phase: take the nearest child of the current node group
            auto node_step = [&]() -> unsigned {
                unsigned fault = 0u;
                const unsigned hitsm = ng.y;
                const unsigned bit = highest_bit(hitsm);
                const unsigned base = ng.x;
                ng.y &= ~(1u << bit);
                if (ng.y > 0x00FFFFFFu && !push(ng)) fault = kErrStackOverflow;
                const unsigned slot = (bit - 24u) ^ octinv;
                const unsigned ci = base + (unsigned)__popc(hitsm & ~(0xFFFFFFFFu << slot));
                if (++steps > p.step_limit) fault |= kErrTimeout;
                if (ci >= (MULTI ? L.node_limit : p.single.node_limit)) fault |= kErrBadScene;
                if (!fault) {
                    const float4* np = L.nodes + (size_t)ci * 5u;
                    const float4 n0 = ld_nc(np + 0), n1 = ld_nc(np + 1), n2 = ld_nc(np + 2);
                    const float4 n3 = ld_nc(np + 3), n4 = ld_nc(np + 4);
                    if (COUNT) ++nvis;
                    const unsigned ew = __float_as_uint(n0.w);
                    const float adjx = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)(ew & 0xFFu) + 127)) << 23), idx_);
                    const float adjy = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)((ew >> 8) & 0xFFu) + 127)) << 23), idy);
                    const float adjz = __fmul_rn(__uint_as_float(((unsigned)((int)(signed char)((ew >> 16) & 0xFFu) + 127)) << 23), idz);
                    const float orx = __fmul_rn(-__fsub_rn(ox, n0.x), idx_);
                    const float ory = __fmul_rn(-__fsub_rn(oy, n0.y), idy);
                    const float orz = __fmul_rn(-__fsub_rn(oz, n0.z), idz);
                    const bool negx = idx_ < 0.f, negy = idy < 0.f, negz = idz < 0.f;
                    const unsigned hitmask = cwbvh_hitmask<ANY>(n1, n2, n3, n4, adjx, adjy, adjz, orx, ory, orz, negx,
                                                           negy, negz, octinv * 0x01010101u, tmin, tmax);
                    ng = make_uint2(__float_as_uint(n1.x), (hitmask & 0xFF000000u) | (ew >> 24));
                    tg = make_uint2(__float_as_uint(n1.y), hitmask & 0x00FFFFFFu);
                }
                return fault;
            };
            unsigned fault = 0u;
            if (active) {
                if (ng.y > 0x00FFFFFFu) {
                    fault = node_step();
                } else {
                    tg = ng;
                    ng = make_uint2(0u, 0u);
                }
                if (fault) finish(fault);
            }
            // Any-hit: lanes whose node produced no triangles and has inner
            // children left descend once more in the same iteration, in the
            // order the next iteration would take, when at least half of the
            // warp would: the second node test costs the warp its full ~285
            // instructions however few lanes take it.  12 scenes / 20M AO
            // rays 3,570 us with it taken for any lane, 3,565 / 3,552 / 3,525
            // / 3,484 / 3,510 / 3,588 us from 4 / 8 / 12 / 16 / 20 / 24 lanes
            // on; 10,592 triangles / 1M rays 220.7 -> 217 us, 8M triangles /
            // 16M rays 5,050 -> 4,976 us.  Taken again while as many lanes
            // would: no gain over once.  Closest-hit loses 1-3 % with any of
            // these limits (its triangle tests, which shrink tmax, get
            // postponed more often).
            if (ANY && __popc(__ballot_sync(kFullMask, active && tg.y == 0u && ng.y > 0x00FFFFFFu)) >= kDeeperMinLanes) {
                if (active && tg.y == 0u && ng.y > 0x00FFFFFFu) {
                    const unsigned f2 = node_step();
                    if (f2) finish(f2);
                }
            }

            // ---- triangle phase, warp-synchronous; postpone when few lanes remain
            {
                const int total = __popc(__ballot_sync(kFullMask, active));
                const int threshold = (int)((float)total * rt);
                for (;;) {
                    const bool want = active && tg.y != 0u;
                    const unsigned wm = __ballot_sync(kFullMask, want);
                    if (wm == 0u) break;
                    if (__popc(wm) < threshold) {
                        if (want && !push(tg)) finish(kErrStackOverflow);
                        break;
                    }
                    if (want) {
                        // Two triangles of the lane's group per round when it
                        // has two, in the group's order: the second is tested
                        // against the tmax the first left, and not at all once
                        // an any-hit ray has finished (fewer warp-wide votes
                        // per triangle: +1.0-2.2 % on single scenes, +1.3 % on
                        // a 64-scene closest-hit batch, +2.0 % on a one-item
                        // batch, +-0.2 % in the ring batch kernel).
                        const unsigned ti = highest_bit(tg.y);
                        const unsigned tri = tg.x * 3u + ti * 3u;
                        tg.y &= ~(1u << ti);
                        const bool two = tg.y != 0u;
                        unsigned tri2 = tri;
                        if (two) {
                            const unsigned ti2 = highest_bit(tg.y);
                            tri2 = tg.x * 3u + ti2 * 3u;
                            tg.y &= ~(1u << ti2);
                        }
                        if (tri >= woop_limit()) {
                            finish(kErrBadScene);
                        } else {
                            const float4* tp = L.woop + tri;
                            if (COUNT) ++ntri;
                            float t, u, v;
                            const float4 v0 = ld_nc(tp), v1 = ld_nc(tp + 1), v2 = ld_nc(tp + 2);
                            if (woop_test(v0, v1, v2, ox, oy, oz, dx, dy, dz, tmin, tmax, t, u, v)) {
                                if (ANY) {
                                    end_ray(t, (int)tri, u, v);
                                } else {
                                    tmax = t;
                                    park_hit((int)tri, u, v);
                                }
                            }
                            if (two && active) {
                                if (tri2 >= woop_limit()) {
                                    finish(kErrBadScene);
                                } else {
                                    const float4* tp2 = L.woop + tri2;
                                    if (COUNT) ++ntri;
                                    const float4 w0 = ld_nc(tp2), w1 = ld_nc(tp2 + 1), w2 = ld_nc(tp2 + 2);
                                    if (woop_test(w0, w1, w2, ox, oy, oz, dx, dy, dz, tmin, tmax, t, u, v)) {
                                        if (ANY) {
                                            end_ray(t, (int)tri2, u, v);
                                        } else {
                                            tmax = t;
                                            park_hit((int)tri2, u, v);
                                        }
                                    }
                                }
                            }
                        }
                    }
                }
            }

            // ---- continue with the stack, or finish the ray
            if (active && ng.y <= 0x00FFFFFFu) {
                if (sp > 0) ng = pop();
                else finish(0u);
            }

            const unsigned am = __ballot_sync(kFullMask, active);
            if (am == 0u) break;
            lost += 32 - __popc(am) - p.fetch_nd;
            if (lost >= p.fetch_nw) break;
        }
    }
    if (RING) cp_async_wait<0>();  // no copy into the ring outlives the block
}

// Launches too small to fill the GPU: one ray per group and no ray counter, the
// grid covers the rays, the group's stack in shared memory.  A node costs the
// warp more issue slots per ray (~130 for 4 rays or ~190 for 8 instead of ~285
// for 32), so a launch that fills the GPU is faster with a lane per ray;
// launch_trace has the measured lines.  10,592 triangles, 4,096 rays, whole AO
// bake 53.4 -> 29.7 us, closest-hit call 50.4 -> 24.7 us.
constexpr int kLanesBlock = 128;

template <bool ANY, bool MULTI, int G>
__global__ void __launch_bounds__(kLanesBlock) cwbvh_lanes_kernel(const TraceParams p) {
    constexpr int kRays = kLanesBlock / G;
    __shared__ uint2 stacks[kRays][kStackTotal];
    const unsigned c = threadIdx.x % G;
    uint2* const stack = stacks[threadIdx.x / G];

    Lane L{};
    float ox = 0.f, oy = 0.f, oz = 0.f, dx = 0.f, dy = 0.f, dz = 0.f, tmin = 0.f, tmax = 0.f;
    float idx_ = 0.f, idy = 0.f, idz = 0.f;
    unsigned octinv = 0;
    uint2 ng = make_uint2(0u, 0x80000000u);
    int sp = 0, hit_addr = -1, steps = 0;
    float hu = 0.f, hv = 0.f;

    const int64_t g = (int64_t)blockIdx.x * kRays + threadIdx.x / G;
    bool active = g < p.total_rays;
    if (active) {
        L.item = -1;
        const Ray r = fetch_ray<MULTI>(p, g, L);
        ox = r.origin_tmin.x; oy = r.origin_tmin.y; oz = r.origin_tmin.z; tmin = r.origin_tmin.w;
        dx = r.dir_tmax.x; dy = r.dir_tmax.y; dz = r.dir_tmax.z; tmax = r.dir_tmax.w;
        idx_ = guarded_rcp(dx);
        idy = guarded_rcp(dy);
        idz = guarded_rcp(dz);
        octinv = 7u - (((dx < 0.f) ? 4u : 0u) | ((dy < 0.f) ? 2u : 0u) | ((dz < 0.f) ? 1u : 0u));
    }
    auto end = [&](int addr) {
        if (c == 0u) finish_ray<MULTI>(p, L, tmax, addr, hu, hv);
        active = false;
    };
    lanes_loop<ANY, G, false>(
        L.nodes, L.woop, L.node_limit, p.step_limit, ox, oy, oz, dx, dy, dz, idx_, idy, idz, octinv, tmin, tmax, ng, sp,
        steps, active, [&]() { return L.woop_limit; },
        [&](uint2 v) {
            if (sp >= kStackTotal) return false;
            if (c == 0u) stack[sp] = v;
            ++sp;
            return true;
        },
        [&]() { return stack[--sp]; },
        [&](float t, int addr, float u, float v) {
            tmax = t;
            hu = u;
            hv = v;
            hit_addr = addr;
            if (ANY) end(addr);
        },
        [&](unsigned err) {
            if (err && c == 0u) atomicOr(&p.scratch->error, err);
            end(err ? -1 : hit_addr);
        });
}

// ------------------------------------------------------------------- BVH2 --

template <bool ANY, int SMEM, bool MULTI, bool COUNT>
__global__ void RQ_BVH2_BOUNDS bvh2_kernel(const TraceParams p) {
    extern __shared__ int istack[];
    constexpr int LOCAL = kStackTotal - SMEM;
    int lstack[LOCAL];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned tid = threadIdx.x;
    const unsigned B = blockDim.x;
    const bool speculate = p.bvh2_speculative != 0;

    Lane L{};
    float ox = 0.f, oy = 0.f, oz = 0.f, dx = 0.f, dy = 0.f, dz = 0.f, tmin = 0.f, tmax = 0.f;
    float idx_ = 0.f, idy = 0.f, idz = 0.f, oodx = 0.f, oody = 0.f, oodz = 0.f;
    int node = 0, leaf = 0, tcur = 0, sp = 0, hit_addr = -1, steps = 0, nvis = 0, ntri = 0;
    float hu = 0.f, hv = 0.f;
    bool active = false, exhausted = false;

    // Stack slot 0 holds the sentinel; entries 1.. are pushed far children.
    auto push = [&](int v) -> bool {
        ++sp;
        if (sp < SMEM) istack[(unsigned)sp * B + tid] = v;
        else if (sp < kStackTotal) lstack[sp - SMEM] = v;
        else { --sp; return false; }
        return true;
    };
    auto pop = [&]() -> int {
        const int v = sp == 0 ? (int)kBvh2Sentinel : (sp < SMEM ? istack[(unsigned)sp * B + tid] : lstack[sp - SMEM]);
        if (sp > 0) --sp;
        return v;
    };
    auto finish = [&](unsigned err) {
        if (err) {
            atomicOr(&p.scratch->error, err);
            hit_addr = -1;
        }
        finish_ray<MULTI>(p, L, tmax, hit_addr, hu, hv);
        if (COUNT) {
            p.node_visits[L.gidx] = nvis;
            p.tri_tests[L.gidx] = ntri;
        }
        active = false;
    };

    for (;;) {
        const bool need = !active && !exhausted;
        const unsigned needm = __ballot_sync(kFullMask, need);
        if (needm) {
            const int leader = __ffs(needm) - 1;
            unsigned long long base = 0;
            if ((int)lane == leader) base = atomicAdd(&p.scratch->ray_counter, (unsigned long long)__popc(needm));
            base = __shfl_sync(kFullMask, base, leader);
            if (need) {
                const int64_t g = (int64_t)base + __popc(needm & lanemask_lt());
                if (g < p.total_rays) {
                    const Ray r = fetch_ray<MULTI>(p, g, L);
                    ox = r.origin_tmin.x; oy = r.origin_tmin.y; oz = r.origin_tmin.z; tmin = r.origin_tmin.w;
                    dx = r.dir_tmax.x; dy = r.dir_tmax.y; dz = r.dir_tmax.z; tmax = r.dir_tmax.w;
                    idx_ = guarded_rcp(dx);
                    idy = guarded_rcp(dy);
                    idz = guarded_rcp(dz);
                    oodx = __fmul_rn(ox, idx_);
                    oody = __fmul_rn(oy, idy);
                    oodz = __fmul_rn(oz, idz);
                    node = 0; leaf = 0; sp = 0; hit_addr = -1; hu = 0.f; hv = 0.f; steps = 0; nvis = 0; ntri = 0;
                    active = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(kFullMask, active) == 0u) break;

        int lost = 0;
        for (;;) {
            // ---- inner-node loop (src/TraversalKernelBVH2.cu:70-122)
            if (active) leaf = 0;
            for (;;) {
                const bool in = active && node != (int)kBvh2Sentinel && node >= 0 && (speculate || leaf >= 0);
                if (__ballot_sync(kFullMask, in) == 0u) break;
                if (in) {
                    unsigned fault = 0u;
                    if (++steps > p.step_limit) fault |= kErrTimeout;
                    if ((unsigned)node >= L.node_limit) fault |= kErrBadScene;
                    if (!fault) {
                        const float4* np = L.nodes + node;
                        const float4 n0 = ld_nc(np), n1 = ld_nc(np + 1), n2 = ld_nc(np + 2), n3 = ld_nc(np + 3);
                        if (COUNT) ++nvis;
                        // Slabs: lo * idir - ood (src/TraversalKernelBVH2.cu:16-19).
                        const float a0lx = __fmaf_rn(n0.x, idx_, -oodx), a0hx = __fmaf_rn(n0.y, idx_, -oodx);
                        const float a0ly = __fmaf_rn(n0.z, idy, -oody), a0hy = __fmaf_rn(n0.w, idy, -oody);
                        const float a0lz = __fmaf_rn(n2.x, idz, -oodz), a0hz = __fmaf_rn(n2.y, idz, -oodz);
                        const float a1lx = __fmaf_rn(n1.x, idx_, -oodx), a1hx = __fmaf_rn(n1.y, idx_, -oodx);
                        const float a1ly = __fmaf_rn(n1.z, idy, -oody), a1hy = __fmaf_rn(n1.w, idy, -oody);
                        const float a1lz = __fmaf_rn(n2.z, idz, -oodz), a1hz = __fmaf_rn(n2.w, idz, -oodz);
                        const float c0min = imin_then_max(a0lz, a0hz, imin_then_max(a0ly, a0hy, imin_then_max(a0lx, a0hx, tmin)));
                        const float c0max = imax_then_min(a0lz, a0hz, imax_then_min(a0ly, a0hy, imax_then_min(a0lx, a0hx, tmax)));
                        const float c1min = imin_then_max(a1lz, a1hz, imin_then_max(a1ly, a1hy, imin_then_max(a1lx, a1hx, tmin)));
                        const float c1max = imax_then_min(a1lz, a1hz, imax_then_min(a1ly, a1hy, imax_then_min(a1lx, a1hx, tmax)));
                        const bool t0 = c0min <= c0max, t1 = c1min <= c1max;
                        int cx = __float_as_int(n3.x), cy = __float_as_int(n3.y);
                        if (!t0 && !t1) {
                            node = pop();
                        } else {
                            node = t0 ? cx : cy;
                            if (t0 && t1) {
                                if (c1min < c0min) { const int tmp = node; node = cy; cy = tmp; }
                                if (!push(cy)) fault |= kErrStackOverflow;
                            }
                        }
                        if (!fault && node < 0 && leaf >= 0) {
                            leaf = node;
                            node = pop();
                        }
                    }
                    if (fault) finish(fault);
                }
                if (speculate && __ballot_sync(kFullMask, in && leaf >= 0) == 0u) break;
            }

            // ---- leaf loop, one triangle per iteration (src/TraversalKernelBVH2.cu:124-169)
            if (active && leaf < 0) tcur = ~leaf;
            for (;;) {
                const bool want = active && leaf < 0;
                if (__ballot_sync(kFullMask, want) == 0u) break;
                if (want) {
                    if ((unsigned)tcur >= L.woop_limit) {
                        finish(kErrBadScene);
                    } else {
                        const float4 v0 = ld_nc(L.woop + tcur);
                        if (__float_as_uint(v0.x) == 0x80000000u) {
                            // Leaf terminator: move to the postponed node / next leaf.
                            leaf = node;
                            if (node < 0) {
                                node = pop();
                                tcur = ~leaf;
                            }
                        } else if (L.woop_limit - (unsigned)tcur < 3u) {
                            finish(kErrBadScene);
                        } else {
                            const float4 v1 = ld_nc(L.woop + tcur + 1), v2 = ld_nc(L.woop + tcur + 2);
                            if (COUNT) ++ntri;
                            float t, u, v;
                            if (woop_test(v0, v1, v2, ox, oy, oz, dx, dy, dz, tmin, tmax, t, u, v)) {
                                tmax = t;
                                hit_addr = tcur;
                                hu = u;
                                hv = v;
                                if (ANY) finish(0u);
                            }
                            tcur += 3;
                        }
                    }
                }
            }

            if (active && node == (int)kBvh2Sentinel) finish(0u);

            const unsigned am = __ballot_sync(kFullMask, active);
            if (am == 0u) break;
            lost += 32 - __popc(am) - p.fetch_nd;
            if (lost >= p.fetch_nw) break;
        }
    }
}

// ---------------------------------------------------------------- launch --

template <bool MULTI, bool COUNT, bool RING>
static TraceKernelFn select_cwbvh(bool any, int smem) {
#define RQ_CW(A, S) (TraceKernelFn)cwbvh_kernel<A, S, MULTI, COUNT, RING>
    if (any) return smem <= 4 ? RQ_CW(true, 4) : (smem <= 8 ? RQ_CW(true, 8) : RQ_CW(true, 16));
    return smem <= 4 ? RQ_CW(false, 4) : (smem <= 8 ? RQ_CW(false, 8) : RQ_CW(false, 16));
#undef RQ_CW
}
template <bool MULTI, bool COUNT>
static TraceKernelFn select_bvh2(bool any, int smem) {
#define RQ_B2(A, S) (TraceKernelFn)bvh2_kernel<A, S, MULTI, COUNT>
    if (any) return smem <= 4 ? RQ_B2(true, 4) : (smem <= 8 ? RQ_B2(true, 8) : RQ_B2(true, 16));
    return smem <= 4 ? RQ_B2(false, 4) : (smem <= 8 ? RQ_B2(false, 8) : RQ_B2(false, 16));
#undef RQ_B2
}

TraceKernelFn trace_kernel(rq_bvh_kind kind, bool any, int smem, bool multi, bool count, bool ring) {
    if (kind == RQ_BVH_CWBVH) {
        if (count) return select_cwbvh<false, true, false>(any, smem);
        if (ring && any && multi) {
            return smem <= 4 ? (TraceKernelFn)cwbvh_kernel<true, 4, true, false, true>
                             : (smem <= 8 ? (TraceKernelFn)cwbvh_kernel<true, 8, true, false, true>
                                          : (TraceKernelFn)cwbvh_kernel<true, 16, true, false, true>);
        }
        if (!multi) return select_cwbvh<false, false, false>(any, smem);
        return select_cwbvh<true, false, false>(any, smem);
    }
    if (count) return select_bvh2<false, true>(any, smem);
    return multi ? select_bvh2<true, false>(any, smem) : select_bvh2<false, false>(any, smem);
}

TraceKernelFn lanes_kernel(bool any, bool multi, int g) {
#define RQ_LN(G) (any ? (multi ? (TraceKernelFn)cwbvh_lanes_kernel<true, true, G> : (TraceKernelFn)cwbvh_lanes_kernel<true, false, G>) \
                      : (multi ? (TraceKernelFn)cwbvh_lanes_kernel<false, true, G> : (TraceKernelFn)cwbvh_lanes_kernel<false, false, G>))
    return g == 8 ? RQ_LN(8) : RQ_LN(4);
#undef RQ_LN
}
int lanes_block() { return kLanesBlock; }

int smem_entries_of(int requested) { return requested <= 4 ? 4 : (requested <= 8 ? 8 : 16); }

size_t trace_smem_bytes(rq_bvh_kind kind, int smem_entries, int block, bool multi, bool ring) {
    if (kind != RQ_BVH_CWBVH) return sizeof(int) * (size_t)smem_entries * (size_t)block;
    return sizeof(uint2) * (size_t)smem_entries * (size_t)block +
           (park_bytes_per_warp(multi) + (ring ? kRingBytesPerWarp : 0)) * (size_t)(block / 32);
}

}  // namespace rq
