// Internal interface between librq's host runtime and its CUDA kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rq.h"

namespace rq {

// Byte-identical to the reference's Ray / Hit (src/helper_math.h:1853-1865).
struct Ray {
    float4 origin_tmin;
    float4 dir_tmax;
};
struct Hit {
    float4 t_triId_u_v;
};
static_assert(sizeof(Ray) == 32 && sizeof(Hit) == 16, "Ray/Hit layout");
static_assert(sizeof(rq_ray) == 32 && sizeof(rq_hit) == 16, "rq_ray/rq_hit layout");

// Error bits a kernel may set in its context's error word.
enum : unsigned {
    kErrStackOverflow = 1u,
    kErrTimeout = 2u,
    kErrBadScene = 4u,
};

// Device scratch of one context: the dynamic-fetch counter and the error word.
constexpr int kDefaultStepLimit = 1 << 22;  // node visits per ray before kErrTimeout (rq_launch.step_limit = 0)

struct DevScratch {
    unsigned long long ray_counter;
    unsigned int error;
    unsigned int pad;
};

// One (scene, rays, hits) unit of work.  Rays [0, count) of this item are the
// global rays [ray_begin, ray_begin + count).  With perm set, ray k is written
// to hits[perm[k]] (the rays were reordered before tracing).
struct TraceItem {
    const float4* nodes;
    const float4* woop;
    const Ray* rays;
    Hit* hits;
    const int32_t* perm;
    int64_t ray_begin;
    int64_t count;
    // Bounds checks: addresses from these on leave the buffers (trace.cu).
    uint32_t node_limit;  // CWBVH: nodes; BVH2: float4 addresses with a whole node behind them
    uint32_t woop_limit;  // CWBVH: addresses with three rows behind them; BVH2: float4 of the buffer
    uint32_t* ao_counts;  // non-null: occluded rays are counted per surfel here instead of writing hits
    int32_t ao_spp;       // rays per surfel (consecutive) when ao_counts is set
    int32_t pad;
};

// Limits of a buffer of f4 float4 (at most UINT32_MAX): whole records in it,
// and addresses with `rows` float4 behind them.  A kernel then checks an
// address with one 32-bit compare instead of a 64-bit sum and compare.
inline uint32_t record_limit(int64_t f4, int64_t record) { return (uint32_t)(f4 / record); }
inline uint32_t address_limit(int64_t f4, int64_t rows) { return f4 >= rows ? (uint32_t)(f4 - rows + 1) : 0u; }

struct TraceParams {
    TraceItem single;         // the scene when the kernel is not a batch kernel
    const TraceItem* items;   // device array of n_items (batch kernels)
    int n_items;
    int64_t total_rays;
    DevScratch* scratch;
    int32_t* node_visits;     // per global ray, counting kernels only
    int32_t* tri_tests;
    float postpone_ratio;
    int fetch_nd;
    int fetch_nw;
    int bvh2_speculative;
    int step_limit;           // node visits per ray before kErrTimeout
};

typedef void (*TraceKernelFn)(TraceParams);

// ring: the CWBVH any-hit batch kernel that prefetches rays into a per-warp
// ring in shared memory (see trace.cu), for batches of at least
// kRingMinRaysPerThread rays per thread of the grid.
constexpr int64_t kRingMinRaysPerThread = 16;
TraceKernelFn trace_kernel(rq_bvh_kind kind, bool any, int smem, bool multi, bool count, bool ring);
// The CWBVH kernel with g = 8 or 4 lanes to a ray for small launches (see
// trace.cu), launched with lanes_block() threads per lanes_block() / g rays.
TraceKernelFn lanes_kernel(bool any, bool multi, int g);
int lanes_block();
int smem_entries_of(int requested);
size_t trace_smem_bytes(rq_bvh_kind kind, int smem_entries, int block, bool multi, bool ring);

}  // namespace rq
