// AO ray generation from a surfel sample cache, surfel sampling on triangles,
// the per-surfel AO reduction and Morton ray sorting.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>

#include "runtime.h"
#include "trace_common.cuh"

namespace rq {

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel Random Numbers: As
// Easy as 1, 2, 3", SC 2011): a counter-based generator, so ray i's numbers
// depend only on (seed, i) and any thread can make them.
struct U4 {
    uint32_t x, y, z, w;
};
__host__ __device__ inline U4 philox4x32_10(U4 c, uint32_t k0, uint32_t k1) {
    constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)M0 * c.x;
        const uint64_t p1 = (uint64_t)M1 * c.z;
        const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
        c = U4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
        k0 += W0;
        k1 += W1;
    }
    return c;
}
// Uniform in (0, 1] from the top 24 bits (curand_uniform's range).
__host__ __device__ inline float unit24(uint32_t r) { return (float)((r >> 8) + 1u) * (1.0f / 16777216.0f); }

__device__ inline float3 f3(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ inline float3 add3(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ inline float3 sub3(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ inline float3 mul3(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ inline float3 cross3(float3 a, float3 b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ inline float len3(float3 a) { return sqrtf(a.x * a.x + a.y * a.y + a.z * a.z); }
__device__ inline float3 norm3(float3 a) { return mul3(a, 1.0f / len3(a)); }

// A whole ray as one 32-byte store (st.v8, sm_100): two 16-byte stores fill
// their sectors by halves and cost the L2 two writes per sector.  `wide`: the
// buffer is 32-byte aligned (the interface asks for 16).
__device__ __forceinline__ void store_ray(Ray* r, float4 o, float4 d, bool wide) {
    if (wide) {
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(r), "f"(o.x), "f"(o.y), "f"(o.z),
                     "f"(o.w), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w)
                     : "memory");
    } else {
        r->origin_tmin = o;
        r->dir_tmax = d;
    }
}
static bool aligned32(const void* p) { return ((uintptr_t)p & 31u) == 0; }

// Surfel frame in shared memory: normal, tangents, ray origin.
struct SurfelFrame {
    float3 n, t1, t2, o;
};

constexpr int kAoBlock = 256;

// One ray per (surfel, sample), surfel = i / spp: tangent frame from n x z
// (n x y when that is short), concentric disk lifted to the cosine
// hemisphere, origin pushed off the surface by radius * offset_scale
// (src/ValidationKernels.cu:41-101).  The random stream of ray i is keyed by
// its index first_ray + i in the whole request, so a request generated in
// pieces gives the same rays as in one call.
//
// Bound by instruction issue (277 warp instructions for 32 rays of 32 B), so
// what a surfel's rays share is computed once: the block's first threads make
// its surfels' frames in shared memory, and the ray threads read them.  A
// block's rays start `skip` samples into its first surfel.  16M rays at 4 per
// surfel 199 -> 159 us, 1M at 32 per surfel 16.6 -> 12.7 us, the same bits.
template <bool SMALL>
__device__ __forceinline__ void aorays_block(
        SurfelFrame* frames, int64_t block, const float4* __restrict__ pos, const float4* __restrict__ nrm,
        const float* __restrict__ radius, int64_t n_rays, FastDiv spp, int64_t first_ray, uint32_t k0, uint32_t k1,
        float tmin, float tmax, float offset_scale, Ray* __restrict__ out, bool wide, uint32_t* __restrict__ counts) {
    const int64_t block0 = block * kAoBlock;
    const int64_t surfel0 = SMALL ? (int64_t)spp.div((uint32_t)block0) : block0 / spp.d;  // SMALL: n_rays < 2^31
    const uint32_t skip = (uint32_t)(block0 - surfel0 * spp.d);
    const uint32_t here = (uint32_t)(n_rays - block0 < kAoBlock ? n_rays - block0 : kAoBlock);  // rays of the block
    // skip < spp and here <= 256, so the sum is below 2^31 + 255.  From 2^31 on
    // the division is past FastDiv's general range but still exact: spp is then
    // above 2^31 - 256, and the quotient 1 far from its ends.
    const uint32_t n_surfels = spp.div(skip + here - 1u) + 1u;
    if (threadIdx.x < n_surfels) {
        const int64_t s = surfel0 + threadIdx.x;
        if (counts && (threadIdx.x > 0 || skip == 0)) counts[s] = 0u;  // the block of a surfel's first ray
        const float3 p = f3(pos[s]);
        const float3 n = f3(nrm[s]);
        const float r = radius ? radius[s] : 0.0f;
        float3 t1 = cross3(n, make_float3(0.f, 0.f, 1.f));
        if (len3(t1) < 0.1f) t1 = cross3(n, make_float3(0.f, 1.f, 0.f));
        t1 = norm3(t1);
        const float3 t2 = norm3(cross3(t1, n));
        SurfelFrame& f = frames[threadIdx.x];
        f.n = n;
        f.t1 = t1;
        f.t2 = t2;
        const bool none = n.x == 0.f && n.y == 0.f && n.z == 0.f;
        f.o = none ? p : add3(p, mul3(n, r * offset_scale));
    }
    __syncthreads();
    if (threadIdx.x >= here) return;
    const int64_t i = block0 + threadIdx.x;
    const SurfelFrame& f = frames[spp.div(skip + threadIdx.x)];
    const float3 n = f.n, o = f.o;
    if (n.x == 0.f && n.y == 0.f && n.z == 0.f) {  // no surface (a primary miss): an empty ray
        store_ray(out + i, make_float4(o.x, o.y, o.z, 0.f), make_float4(0.f, 0.f, 1.f, 0.f), wide);
        return;
    }
    const uint64_t ctr = (uint64_t)(first_ray + i);
    const U4 rnd = philox4x32_10(U4{(uint32_t)ctr, (uint32_t)(ctr >> 32), 0u, 0u}, k0, k1);
    const float a = 2.0f * unit24(rnd.x) - 1.0f, b = 2.0f * unit24(rnd.y) - 1.0f;
    float dxl = 0.f, dyl = 0.f;
    if (a != 0.f || b != 0.f) {
        const float kPi = 3.1415926f;
        const bool x_major = a * a > b * b;
        const float rr = x_major ? a : b;
        const float q = (x_major ? b : a) / rr;
        const float th = x_major ? __fmul_rn(kPi / 4.0f, q) : __fmaf_rn(-(kPi / 4.0f), q, kPi / 2.0f);
        float sn, cs;
        sincosf(th, &sn, &cs);
        dxl = rr * cs;
        dyl = rr * sn;
    }
    const float dzl = sqrtf(fmaxf(0.0f, 1.0f - dxl * dxl - dyl * dyl));
    const float3 d = norm3(add3(add3(mul3(f.t1, dxl), mul3(f.t2, dyl)), mul3(n, dzl)));
    store_ray(out + i, make_float4(o.x, o.y, o.z, tmin), make_float4(d.x, d.y, d.z, tmax), wide);
}

template <bool SMALL>
__global__ void __launch_bounds__(kAoBlock) aorays_kernel(
        const float4* __restrict__ pos, const float4* __restrict__ nrm, const float* __restrict__ radius,
        int64_t n_rays, FastDiv spp, int64_t first_ray, uint32_t k0, uint32_t k1, float tmin, float tmax,
        float offset_scale, Ray* __restrict__ out, bool wide) {
    __shared__ SurfelFrame frames[kAoBlock];
    aorays_block<SMALL>(frames, blockIdx.x, pos, nrm, radius, n_rays, spp, first_ray, k0, k1, tmin, tmax, offset_scale,
                        out, wide, nullptr);
}

// The pieces of a bake launch together: a block finds its piece by its number.
template <class Begin>
__device__ __forceinline__ int item_of_block(const AoItem* items, int n_items, Begin begin) {
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (begin(items[mid]) <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kAoBlock) aorays_items_kernel(const AoItem* __restrict__ items, int n_items) {
    __shared__ SurfelFrame frames[kAoBlock];
    const AoItem& it = items[item_of_block(items, n_items, [](const AoItem& i) { return i.block_begin; })];
    aorays_block<true>(frames, blockIdx.x - it.block_begin, it.pos, it.nrm, it.radius, it.n_rays, it.spp, it.first_ray,
                       it.k0, it.k1, it.tmin, it.tmax, it.offset_scale, it.rays, it.wide != 0u, it.counts);
}

// Occluded-ray counts turned into AO fractions (at the counters themselves or
// in mapped host memory).
__global__ void __launch_bounds__(kAoBlock) ao_finish_items_kernel(const AoItem* __restrict__ items, int n_items) {
    const AoItem& it = items[item_of_block(items, n_items, [](const AoItem& i) { return i.surfel_block_begin; })];
    const int64_t i = (int64_t)(blockIdx.x - it.surfel_block_begin) * kAoBlock + threadIdx.x;
    if (i < it.n_surfels) it.ao[i] = (float)it.counts[i] / (float)(int)it.spp.d;
}

// Surfel i on triangle floor(u * nt) at barycentrics (1 - sqrt(a), b sqrt(a)).
__global__ void surfels_kernel(const float* __restrict__ v, const int32_t* __restrict__ idx, int64_t nt,
                               int64_t n, uint32_t k0, uint32_t k1, float4* __restrict__ pos,
                               float4* __restrict__ nrm, float* __restrict__ radius) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const U4 rnd = philox4x32_10(U4{(uint32_t)i, (uint32_t)((uint64_t)i >> 32), 1u, 0u}, k0, k1);
    const uint64_t pick = ((uint64_t)rnd.x << 32 | rnd.y);
    const int64_t t = (int64_t)(((unsigned __int128)pick * (unsigned __int128)nt) >> 64);
    const float su = sqrtf(unit24(rnd.z)), bv = unit24(rnd.w);
    const float b0 = 1.0f - su, b1 = bv * su, b2 = 1.0f - b0 - b1;
    const int32_t* tri = idx + 3 * t;
    const float3 p0 = make_float3(v[3 * tri[0]], v[3 * tri[0] + 1], v[3 * tri[0] + 2]);
    const float3 p1 = make_float3(v[3 * tri[1]], v[3 * tri[1] + 1], v[3 * tri[1] + 2]);
    const float3 p2 = make_float3(v[3 * tri[2]], v[3 * tri[2] + 1], v[3 * tri[2] + 2]);
    const float3 p = add3(add3(mul3(p0, b0), mul3(p1, b1)), mul3(p2, b2));
    const float3 nn = norm3(cross3(sub3(p1, p0), sub3(p2, p0)));
    pos[i] = make_float4(p.x, p.y, p.z, 1.0f);
    nrm[i] = make_float4(nn.x, nn.y, nn.z, 0.0f);
    if (radius) radius[i] = 0.0f;
}

// Pinhole camera: pixel (x, y) centre through an image plane at distance 1.
// Ray i is pixel (x, y) of tile i / (tw * th), tiles row-major across the
// image and pixels row-major within a tile (tw = width, th = 1: the image
// row-major).
//
// Bound by the 32 B written per ray: 4.2M rays 36.6 -> 21.3 us (6.3 TB/s) with
// whole-sector stores.  The four divisions that place a pixel are
// multiplications (FastDiv); images of 2^31 pixels and more divide.
template <bool SMALL>
__global__ void camera_rays_kernel(float3 eye, float3 fwd, float3 right, float3 upv, float half_w, float half_h,
                                   int width, int height, int tw, int th, FastDiv per_tile, FastDiv tiles_x,
                                   FastDiv tile_w, float tmin, float tmax, Ray* __restrict__ out,
                                   bool wide) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)width * height) return;
    int tile_x, tile_y, in_x, in_y;
    if (SMALL) {
        const uint32_t tile = per_tile.div((uint32_t)i), in_tile = (uint32_t)i - tile * per_tile.d;
        const uint32_t ty = tiles_x.div(tile), iy = tile_w.div(in_tile);
        tile_x = (int)(tile - ty * tiles_x.d);
        tile_y = (int)ty;
        in_x = (int)(in_tile - iy * tile_w.d);
        in_y = (int)iy;
    } else {
        const int64_t tile = i / ((int64_t)tw * th), in_tile = i - tile * ((int64_t)tw * th);
        const int across = width / tw;
        tile_x = (int)(tile % across);
        tile_y = (int)(tile / across);
        in_x = (int)(in_tile % tw);
        in_y = (int)(in_tile / tw);
    }
    const int x = tile_x * tw + in_x;
    const int y = tile_y * th + in_y;
    const float sx = ((x + 0.5f) / width * 2.0f - 1.0f) * half_w;
    const float sy = (1.0f - (y + 0.5f) / height * 2.0f) * half_h;
    const float3 d = norm3(add3(add3(fwd, mul3(right, sx)), mul3(upv, sy)));
    store_ray(out + i, make_float4(eye.x, eye.y, eye.z, tmin), make_float4(d.x, d.y, d.z, tmax), wide);
}

// Hit point and facing geometric normal of each closest hit.
__global__ void surfels_from_hits_kernel(const Ray* __restrict__ rays, const Hit* __restrict__ hits,
                                         const float4* __restrict__ woop, int64_t woop_f4, int64_t n,
                                         float4* __restrict__ pos, float4* __restrict__ nrm,
                                         float* __restrict__ radius) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 o = rays[i].origin_tmin, d = rays[i].dir_tmax;
    const float4 h = hits[i].t_triId_u_v;
    const int addr = __float_as_int(h.y);
    if (addr < 0 || addr >= woop_f4) {
        pos[i] = make_float4(o.x, o.y, o.z, 1.0f);
        nrm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        const float4 v0 = __ldg(woop + addr);  // V0 = triangle-space z row: normal to the triangle
        float3 nn = norm3(make_float3(v0.x, v0.y, v0.z));
        if (nn.x * d.x + nn.y * d.y + nn.z * d.z > 0.f) nn = mul3(nn, -1.0f);
        pos[i] = make_float4(o.x + h.x * d.x, o.y + h.x * d.y, o.z + h.x * d.z, 1.0f);
        nrm[i] = make_float4(nn.x, nn.y, nn.z, 0.f);
    }
    if (radius) radius[i] = 0.0f;
}

// Fraction of a surfel's spp rays whose hit id is not -1.  A memory-bound sum:
// P lanes (the largest power of two that leaves each four hits, at most 32)
// take a surfel's hits side by side, four loads in flight each, and add up:
// 16M hits at 32 per surfel 63.8 -> 39.2 us (6.5 TB/s of the hits' sectors),
// 128 surfels 4.1 -> 2 us; a thread per surfel below 8 rays as before.
template <int P>
__global__ void ao_reduce_kernel(const Hit* __restrict__ hits, int64_t n_surfels, int spp, float* __restrict__ ao) {
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x / P) + threadIdx.x / P;
    const unsigned c = threadIdx.x % P, n = (unsigned)spp;
    int occ = 0;
    if (s < n_surfels)
#pragma unroll 4
        for (unsigned k = c; k < n; k += P)  // unsigned: k ends up to P - 1 past spp, which may be past INT_MAX
            occ += __float_as_int(hits[s * spp + k].t_triId_u_v.y) != -1;
#pragma unroll
    for (int m = P / 2; m > 0; m >>= 1) occ += __shfl_xor_sync(kFullMask, occ, m);
    if (c == 0 && s < n_surfels) ao[s] = (float)occ / (float)spp;
}

// ----------------------------------------------------------------- sorting

__device__ inline uint32_t spread10(uint32_t x) {
    x &= 0x3FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// 30-bit ray key: 3 x 9-bit Morton code of the origin inside the bounds
// b (high 27 bits) then the direction octant (low 3 bits).
constexpr int kRayKeyBits = 30;
__device__ inline uint32_t ray_key(const float4& o, const float4& d, const float* b) {
    uint32_t q[3];
    const float oo[3] = {o.x, o.y, o.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float ext = b[3 + a] - b[a];
        float f = ext > 0.f ? (oo[a] - b[a]) / ext : 0.f;
        f = fminf(fmaxf(f, 0.f), 1.f);
        q[a] = min(511u, (uint32_t)(f * 512.0f));
    }
    const uint32_t m = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
    const uint32_t oct = (d.x < 0.f ? 4u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 1u : 0u);
    return (m << 3) | oct;
}

// Keys of the rays of several items: the item number sits above the ray key,
// so every item's rays stay together.
__global__ void morton_keys_kernel(const TraceItem* __restrict__ items, int n_items, const float* __restrict__ bounds,
                                   int64_t total, uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].ray_begin <= g) lo = mid; else hi = mid - 1;
    }
    const TraceItem& it = items[lo];
    const int64_t k = g - it.ray_begin;
    keys[g] = ((uint64_t)lo << 32) | ray_key(it.rays[k].origin_tmin, it.rays[k].dir_tmax, bounds + 6 * lo);
    vals[g] = (int32_t)k;
}

__global__ void gather_rays_kernel(const TraceItem* __restrict__ items, const uint64_t* __restrict__ keys,
                                   const int32_t* __restrict__ vals, int64_t total, Ray* __restrict__ sorted) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const int item = (int)(keys[g] >> 32);
    const Ray* src = items[item].rays + vals[g];
    sorted[g].origin_tmin = __ldg(&src->origin_tmin);
    sorted[g].dir_tmax = __ldg(&src->dir_tmax);
}

// The same for one ray buffer: 32-bit keys (four radix passes of 8-byte pairs
// instead of five of 12), bounds in the launch arguments, and rays moved as
// one 32-byte load and store each (`wide`: both buffers 32-byte aligned).
// Both kernels are bound by their bytes; the gather reads its rays in Morton
// order, a sector at a time, and keeps four of them in flight per thread.
struct Bounds6 {
    float b[6];
};

__device__ __forceinline__ void load_ray(const Ray* r, float4& o, float4& d, bool wide) {
    if (wide) {
        asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w), "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
            : "l"(r));
    } else {
        o = __ldg(&r->origin_tmin);
        d = __ldg(&r->dir_tmax);
    }
}

__global__ void ray_keys_kernel(const Ray* __restrict__ rays, Bounds6 bounds, int64_t n, uint32_t* __restrict__ keys,
                                int32_t* __restrict__ vals, bool wide) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    float4 o, d;
    load_ray(rays + g, o, d, wide);
    keys[g] = ray_key(o, d, bounds.b);
    vals[g] = (int32_t)g;
}

constexpr int kGatherRays = 4;
__global__ void permute_rays_kernel(const Ray* __restrict__ rays, const int32_t* __restrict__ perm, int64_t n,
                                    Ray* __restrict__ sorted, bool wide_in, bool wide_out) {
    const int64_t base = (int64_t)blockIdx.x * (blockDim.x * kGatherRays) + threadIdx.x;
    float4 o[kGatherRays], d[kGatherRays];
#pragma unroll
    for (int q = 0; q < kGatherRays; ++q) {
        const int64_t g = base + (int64_t)q * blockDim.x;
        if (g < n) load_ray(rays + perm[g], o[q], d[q], wide_in);
    }
#pragma unroll
    for (int q = 0; q < kGatherRays; ++q) {
        const int64_t g = base + (int64_t)q * blockDim.x;
        if (g < n) store_ray(sorted + g, o[q], d[q], wide_out);
    }
}

static unsigned blocks_for(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

rq_status aorays_launch(const float* pos, const float* nrm, const float* radius, int64_t n_surfels, int spp,
                        int64_t first_ray, uint64_t seed, float tmin, float tmax, float offset_scale, rq_ray* out_rays,
                        void* stream) {
    if (n_surfels < 0 || spp <= 0 || first_ray < 0 || (n_surfels > 0 && (!pos || !nrm || !out_rays)))
        return RQ_ERR_INVALID_ARG;
    const int64_t n = n_surfels * spp;
    if (n == 0) return RQ_OK;
    const auto kernel = n < ((int64_t)1 << 31) ? aorays_kernel<true> : aorays_kernel<false>;
    kernel<<<blocks_for(n, kAoBlock), kAoBlock, 0, (cudaStream_t)stream>>>(
        (const float4*)pos, (const float4*)nrm, radius, n, FastDiv((uint32_t)spp), first_ray, (uint32_t)seed, (uint32_t)(seed >> 32),
        tmin, tmax, offset_scale, (Ray*)out_rays, aligned32(out_rays));
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

uint32_t ao_ray_blocks(int64_t n_rays) { return blocks_for(n_rays, kAoBlock); }
uint32_t ao_surfel_blocks(int64_t n_surfels) { return blocks_for(n_surfels, kAoBlock); }

rq_status aorays_items_launch(const AoItem* items, int n_items, uint32_t blocks, cudaStream_t s) {
    if (blocks == 0) return RQ_OK;
    aorays_items_kernel<<<blocks, kAoBlock, 0, s>>>(items, n_items);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

rq_status ao_finish_items_launch(const AoItem* items, int n_items, uint32_t blocks, cudaStream_t s) {
    if (blocks == 0) return RQ_OK;
    ao_finish_items_kernel<<<blocks, kAoBlock, 0, s>>>(items, n_items);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

rq_status sort_plan_create(const std::vector<TraceItem>& items, const std::vector<float>& bounds, SortPlan& plan) {
    plan = SortPlan();
    plan.n_items = (int)items.size();
    std::vector<TraceItem> src = items;
    int64_t off = 0;
    for (auto& it : src) {
        it.ray_begin = off;
        off += it.count;
    }
    plan.total = off;
    int bits = 1;
    while ((1 << bits) < plan.n_items) ++bits;
    plan.end_bit = 32 + bits;
    if (plan.total == 0) return RQ_OK;
    const size_t n = (size_t)plan.total;
    RQ_CUDA(cudaMalloc(&plan.keys_in, n * 8));
    RQ_CUDA(cudaMalloc(&plan.keys_out, n * 8));
    RQ_CUDA(cudaMalloc(&plan.vals_in, n * 4));
    RQ_CUDA(cudaMalloc(&plan.vals_out, n * 4));
    RQ_CUDA(cudaMalloc(&plan.sorted, n * sizeof(Ray)));
    RQ_CUDA(cudaMalloc(&plan.src_items, src.size() * sizeof(TraceItem)));
    RQ_CUDA(cudaMemcpy(plan.src_items, src.data(), src.size() * sizeof(TraceItem), cudaMemcpyHostToDevice));
    RQ_CUDA(cudaMalloc(&plan.bounds, bounds.size() * sizeof(float)));
    RQ_CUDA(cudaMemcpy(plan.bounds, bounds.data(), bounds.size() * sizeof(float), cudaMemcpyHostToDevice));
    RQ_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, plan.cub_temp_bytes, plan.keys_in, plan.keys_out, plan.vals_in,
                                            plan.vals_out, (int64_t)n, 0, plan.end_bit));
    RQ_CUDA(cudaMalloc(&plan.cub_temp, std::max<size_t>(16, plan.cub_temp_bytes)));
    // Count the kernels of one sort by capturing it once (not executed).
    cudaStream_t cs;
    RQ_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
        sort_plan_run(plan, cs);
        if (cudaStreamEndCapture(cs, &g) == cudaSuccess && g) {
            size_t n = 0;
            cudaGraphGetNodes(g, nullptr, &n);
            std::vector<cudaGraphNode_t> nodes(n);
            cudaGraphGetNodes(g, nodes.data(), &n);
            for (auto nd : nodes) {
                cudaGraphNodeType t;
                if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) ++plan.n_kernels;
            }
            cudaGraphDestroy(g);
        }
    }
    cudaGetLastError();
    cudaStreamDestroy(cs);
    return RQ_OK;
}

int sort_plan_kernel_count(const SortPlan& plan) { return plan.n_kernels; }

rq_status sort_plan_run(SortPlan& plan, cudaStream_t s) {
    if (plan.total == 0) return RQ_OK;
    morton_keys_kernel<<<blocks_for(plan.total, 256), 256, 0, s>>>(plan.src_items, plan.n_items, plan.bounds,
                                                                   plan.total, plan.keys_in, plan.vals_in);
    RQ_CUDA(cudaGetLastError());
    size_t tb = plan.cub_temp_bytes;
    RQ_CUDA(cub::DeviceRadixSort::SortPairs(plan.cub_temp, tb, plan.keys_in, plan.keys_out, plan.vals_in,
                                            plan.vals_out, plan.total, 0, plan.end_bit, s));
    gather_rays_kernel<<<blocks_for(plan.total, 256), 256, 0, s>>>(plan.src_items, plan.keys_out, plan.vals_out,
                                                                   plan.total, plan.sorted);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

void sort_plan_destroy(SortPlan& plan) {
    cudaFree(plan.keys_in);
    cudaFree(plan.keys_out);
    cudaFree(plan.vals_in);
    cudaFree(plan.vals_out);
    cudaFree(plan.sorted);
    cudaFree(plan.src_items);
    cudaFree(plan.bounds);
    cudaFree(plan.cub_temp);
    plan = SortPlan();
}

}  // namespace rq

using namespace rq;

extern "C" {

rq_status rq_aorays(const float* pos, const float* nrm, const float* radius, int64_t n_surfels, int spp, uint64_t seed,
                    float tmin, float tmax, float offset_scale, rq_ray* out_rays, void* stream) {
    return rq::aorays_launch(pos, nrm, radius, n_surfels, spp, 0, seed, tmin, tmax, offset_scale, out_rays, stream);
}

rq_status rq_sample_surfels(const float* vertices, const int32_t* indices, int64_t nt, int64_t n_surfels,
                            uint64_t seed, float* out_pos, float* out_nrm, float* out_radius, void* stream) {
    if (nt <= 0 || n_surfels < 0 || !vertices || !indices || (n_surfels > 0 && (!out_pos || !out_nrm)))
        return RQ_ERR_INVALID_ARG;
    if (n_surfels == 0) return RQ_OK;
    surfels_kernel<<<blocks_for(n_surfels, 256), 256, 0, (cudaStream_t)stream>>>(
        vertices, indices, nt, n_surfels, (uint32_t)seed, (uint32_t)(seed >> 32), (float4*)out_pos, (float4*)out_nrm,
        out_radius);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

static rq_status camera_rays_impl(const float eye[3], const float look[3], const float up[3], float vfov_deg,
                                  int width, int height, int tw, int th, float tmin, float tmax, rq_ray* out_rays,
                                  void* stream) {
    if (!eye || !look || !up || width <= 0 || height <= 0 || !(vfov_deg > 0.f && vfov_deg < 180.f) || !out_rays)
        return RQ_ERR_INVALID_ARG;
    if (tw <= 0 || th <= 0 || width % tw != 0 || height % th != 0) return RQ_ERR_INVALID_ARG;
    // Camera frame on the host (once per call).
    auto norm = [](float3 a) {
        const float l = std::sqrt(a.x * a.x + a.y * a.y + a.z * a.z);
        return make_float3(a.x / l, a.y / l, a.z / l);
    };
    auto cross = [](float3 a, float3 b) {
        return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
    };
    auto len = [](float3 a) { return std::sqrt(a.x * a.x + a.y * a.y + a.z * a.z); };
    const float3 e = make_float3(eye[0], eye[1], eye[2]);
    const float3 view = make_float3(look[0] - eye[0], look[1] - eye[1], look[2] - eye[2]);
    if (!(len(view) > 0.f) || !std::isfinite(len(view))) return RQ_ERR_INVALID_ARG;
    const float3 fwd = norm(view);
    const float3 side = cross(fwd, make_float3(up[0], up[1], up[2]));
    if (!(len(side) > 1e-6f) || !std::isfinite(len(side))) return RQ_ERR_INVALID_ARG;  // up parallel to the view
    const float3 right = norm(side);
    const float3 upv = cross(right, fwd);
    const float half_h = std::tan(vfov_deg * 0.5f * 3.14159265358979f / 180.0f);
    const float half_w = half_h * (float)width / (float)height;
    const int64_t n = (int64_t)width * height;
    const bool small = n < ((int64_t)1 << 31);
    const FastDiv per_tile(small ? (uint32_t)(tw * th) : 1u), tiles_x((uint32_t)(width / tw)), tile_w((uint32_t)tw);
    const auto kernel = small ? camera_rays_kernel<true> : camera_rays_kernel<false>;
    kernel<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(e, fwd, right, upv, half_w, half_h, width, height,
                                                                 tw, th, per_tile, tiles_x, tile_w, tmin, tmax,
                                                                 (Ray*)out_rays, aligned32(out_rays));
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

rq_status rq_camera_rays(const float eye[3], const float look[3], const float up[3], float vfov_deg, int width,
                         int height, float tmin, float tmax, rq_ray* out_rays, void* stream) {
    return camera_rays_impl(eye, look, up, vfov_deg, width, height, width, 1, tmin, tmax, out_rays, stream);
}

rq_status rq_camera_rays_tiled(const float eye[3], const float look[3], const float up[3], float vfov_deg,
                               int width, int height, int tile_w, int tile_h, float tmin, float tmax,
                               rq_ray* out_rays, void* stream) {
    return camera_rays_impl(eye, look, up, vfov_deg, width, height, tile_w, tile_h, tmin, tmax, out_rays, stream);
}

rq_status rq_surfels_from_hits(rq_scene_t scene, const rq_ray* rays, const rq_hit* hits, int64_t count,
                               float* out_pos, float* out_nrm, float* out_radius, void* stream) {
    if (!scene || count < 0 || (count > 0 && (!rays || !hits || !out_pos || !out_nrm))) return RQ_ERR_INVALID_ARG;
    if (count == 0) return RQ_OK;
    surfels_from_hits_kernel<<<blocks_for(count, 256), 256, 0, (cudaStream_t)stream>>>(
        (const Ray*)rays, (const Hit*)hits, scene->woop, scene->woop_f4, count, (float4*)out_pos, (float4*)out_nrm,
        out_radius);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

rq_status rq_ao_reduce(const rq_hit* hits, int64_t n_surfels, int spp, float* out_ao, void* stream) {
    if (n_surfels < 0 || spp <= 0 || (n_surfels > 0 && (!hits || !out_ao))) return RQ_ERR_INVALID_ARG;
    if (n_surfels == 0) return RQ_OK;
    int lanes = 1;
    while (lanes < 32 && 8 * lanes <= spp) lanes *= 2;
    const auto kernel = lanes == 32 ? ao_reduce_kernel<32> : lanes == 16 ? ao_reduce_kernel<16>
                      : lanes == 8 ? ao_reduce_kernel<8> : lanes == 4 ? ao_reduce_kernel<4>
                      : lanes == 2 ? ao_reduce_kernel<2> : ao_reduce_kernel<1>;
    kernel<<<blocks_for(n_surfels * lanes, 256), 256, 0, (cudaStream_t)stream>>>((const Hit*)hits, n_surfels, spp,
                                                                                 out_ao);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

// The buffers of a sort are kept with the context between calls up to
// kSortKeepBytes (about 20M rays; allocating them, and counting a plan's
// kernels, cost ten times the sort), and given back with it; a larger sort
// allocates its own.  The call ends with its stream synchronized, so the next
// one finds them free; calls on one context from several threads take turns.
constexpr size_t kSortKeepBytes = (size_t)256 << 20;

rq_status rq_sort_rays(rq_ctx_t ctx, const rq_ray* rays, int64_t count, const float bounds_lo[3],
                       const float bounds_hi[3], rq_ray* sorted_rays, int32_t* perm, void* stream) {
    if (!ctx || count < 0 || (count > 0 && (!rays || !sorted_rays || !perm || !bounds_lo || !bounds_hi)))
        return RQ_ERR_INVALID_ARG;
    if (count == 0) return RQ_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t n = (size_t)count;
    // Outputs that overlap the input or each other, or that the kernels' stores
    // are too wide for (rays 16 bytes, numbers 4), are written last, from copies.
    auto overlap = [](const void* a, size_t an, const void* b, size_t bn) {
        return (uintptr_t)a < (uintptr_t)b + bn && (uintptr_t)b < (uintptr_t)a + an;
    };
    const bool staged = overlap(rays, n * sizeof(Ray), sorted_rays, n * sizeof(Ray)) ||
                        overlap(rays, n * sizeof(Ray), perm, n * 4) ||
                        overlap(sorted_rays, n * sizeof(Ray), perm, n * 4) ||
                        ((uintptr_t)sorted_rays & 15u) != 0 || ((uintptr_t)perm & 3u) != 0;
    size_t cub_bytes = 0;
    RQ_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                            (const int32_t*)nullptr, (int32_t*)nullptr, count, 0, kRayKeyBits, s));
    size_t bytes = 0;
    auto take = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t keys_in = take(n * 4), keys_out = take(n * 4), vals_in = take(n * 4), cub_temp = take(cub_bytes);
    const size_t st_rays = staged ? take(n * sizeof(Ray)) : 0, st_perm = staged ? take(n * 4) : 0;

    std::lock_guard<std::mutex> lk(ctx->temp_mu);
    int dev = 0;
    RQ_CUDA(cudaGetDevice(&dev));
    char* base = nullptr;
    const bool keep = bytes <= kSortKeepBytes && dev == ctx->device;
    if (keep) {
        if (ctx->temp_bytes < bytes) {
            cudaFree(ctx->temp);
            ctx->temp = nullptr;
            ctx->temp_bytes = 0;
            RQ_CUDA(cudaMalloc(&ctx->temp, bytes));
            ctx->temp_bytes = bytes;
        }
        base = (char*)ctx->temp;
    } else {
        RQ_CUDA(cudaMalloc(&base, bytes));
    }
    int32_t* const out_perm = staged ? (int32_t*)(base + st_perm) : perm;
    Ray* const out_rays = staged ? (Ray*)(base + st_rays) : (Ray*)sorted_rays;
    const Bounds6 b{{bounds_lo[0], bounds_lo[1], bounds_lo[2], bounds_hi[0], bounds_hi[1], bounds_hi[2]}};
    ray_keys_kernel<<<blocks_for(count, 256), 256, 0, s>>>((const Ray*)rays, b, count, (uint32_t*)(base + keys_in),
                                                           (int32_t*)(base + vals_in), aligned32(rays));
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cub::DeviceRadixSort::SortPairs(base + cub_temp, cub_bytes, (const uint32_t*)(base + keys_in),
                                            (uint32_t*)(base + keys_out), (const int32_t*)(base + vals_in), out_perm,
                                            count, 0, kRayKeyBits, s);
    if (e == cudaSuccess) {
        permute_rays_kernel<<<blocks_for(count, 256 * kGatherRays), 256, 0, s>>>(
            (const Ray*)rays, out_perm, count, out_rays, aligned32(rays), aligned32(out_rays));
        e = cudaGetLastError();
    }
    if (staged && e == cudaSuccess)
        e = cudaMemcpyAsync(sorted_rays, out_rays, n * sizeof(Ray), cudaMemcpyDeviceToDevice, s);
    if (staged && e == cudaSuccess) e = cudaMemcpyAsync(perm, out_perm, n * 4, cudaMemcpyDeviceToDevice, s);
    const cudaError_t done = cudaStreamSynchronize(s);  // also after an error: the buffers are reused or freed
    if (e == cudaSuccess) e = done;
    if (!keep) cudaFree(base);
    return e == cudaSuccess ? RQ_OK : cuda_fail(e, "rq_sort_rays");
}

}  // extern "C"
