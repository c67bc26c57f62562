// Internal runtime objects behind the C ABI handles.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "device_api.h"

struct rq_ctx {
    int device = 0;
    rq::DevScratch* scratch = nullptr;  // device
    void* temp = nullptr;               // sort buffers kept between rq_sort_rays calls
    size_t temp_bytes = 0;
    std::mutex temp_mu;                 // held by a call that uses them
};

struct rq_scene {
    rq_bvh_kind kind;
    int device = 0;
    const float4* nodes = nullptr;
    const float4* woop = nullptr;
    const int32_t* prim_index = nullptr;
    int64_t node_f4 = 0, woop_f4 = 0, prim_count = 0;
    bool owned = false;
    void* block = nullptr;   // the one allocation the owned buffers lie in (null: one each)
    cudaEvent_t scratch_freed = nullptr;  // built on the device, holds its build scratch pool: behind the scratch's frees
    float lo[3] = {0.f, 0.f, 0.f};
    float hi[3] = {0.f, 0.f, 0.f};
};

namespace rq {

// Records a failing CUDA call for rq_last_error and maps it to a status.
rq_status cuda_fail(cudaError_t e, const char* what);
// Sets the text rq_last_error returns on this thread.
void set_last_error(const std::string& msg);

#define RQ_CUDA(call)                                          \
    do {                                                       \
        cudaError_t rq_e_ = (call);                            \
        if (rq_e_ != cudaSuccess) return rq::cuda_fail(rq_e_, #call); \
    } while (0)

int device_sms(int device);

// A scene that rq_build_scene_gpu made on `device` was destroyed (gpubuild.cu);
// takes its event.
void gpu_built_scene_gone(int device, cudaEvent_t scratch_freed);

// Fills zero fields of `l` with defaults for this BVH kind / query.
rq_launch resolve_launch(rq_bvh_kind kind, rq_query q, const rq_launch* l);

// Launches the trace kernel for p's rays (and zeroes the ray counter for the
// persistent ones).  With the default launch shape, small CWBVH launches take
// the kernel with several lanes to a ray.
rq_status launch_trace(rq_bvh_kind kind, rq_query q, const rq_launch& l, bool multi, bool count,
                       const TraceParams& p, cudaStream_t s);

// Computes the occupancy of a kernel variant ahead of a stream capture.
void warm_launch_cache(rq_bvh_kind kind, rq_query q, const rq_launch& l, bool multi, bool count);

// Zeroes the context's ray counter on the stream.
rq_status reset_counter(rq_ctx* ctx, cudaStream_t s);

TraceItem scene_item(const rq_scene* sc, const rq_ray* rays, rq_hit* hits, int64_t count);
TraceParams base_params(rq_ctx* ctx, const rq_launch& l);

// AO rays of n_surfels surfels (rays.cu); ray k of the call is ray
// first_ray + k of the request it belongs to (its random stream).
rq_status aorays_launch(const float* pos, const float* nrm, const float* radius, int64_t n_surfels, int spp,
                        int64_t first_ray, uint64_t seed, float tmin, float tmax, float offset_scale, rq_ray* out_rays,
                        void* stream);

// Division of 31-bit numbers by one divisor: floor(i / d) = i * mul >> shift
// with mul = ceil(2^shift / d) and shift = 31 + ceil(log2 d) is exact for every
// i < 2^31 (Granlund and Montgomery, "Division by Invariant Integers using
// Multiplication", PLDI 1994), mul < 2^32.
struct FastDiv {
    uint32_t mul, shift, d;
    explicit FastDiv(uint32_t divisor) : d(divisor) {
        uint32_t l = 0;
        while (l < 31 && (1ull << l) < divisor) ++l;
        shift = 31 + l;
        mul = (uint32_t)(((1ull << shift) + divisor - 1) / divisor);
    }
    __device__ uint32_t div(uint32_t i) const { return (uint32_t)((uint64_t)i * mul >> shift); }
};

// AO bake work of one launch over several pieces (rays.cu): piece k's rays are
// made by blocks [block_begin, next piece's), which also zero its counters;
// the counters then become AO fractions at `ao`.  Inputs and `ao` are device
// addresses, of device memory or of mapped host memory.
struct AoItem {
    const float4* pos;
    const float4* nrm;
    const float* radius;
    Ray* rays;
    uint32_t* counts;
    float* ao;
    int64_t first_ray;
    int64_t n_surfels;
    FastDiv spp;
    uint32_t n_rays;  // below 2^31
    uint32_t k0, k1;
    float tmin, tmax, offset_scale;
    uint32_t block_begin;         // of the ray launch
    uint32_t surfel_block_begin;  // of the AO launch
    uint32_t wide;                // rays 32-byte aligned
};
uint32_t ao_ray_blocks(int64_t n_rays);      // blocks of a piece in the ray launch
uint32_t ao_surfel_blocks(int64_t n_surfels);  // and in the AO launch
rq_status aorays_items_launch(const AoItem* items, int n_items, uint32_t blocks, cudaStream_t s);
rq_status ao_finish_items_launch(const AoItem* items, int n_items, uint32_t blocks, cudaStream_t s);

// Morton keys + radix sort of the rays of several items (rays.cu).
struct SortPlan {
    int n_items = 0;
    int64_t total = 0;
    // device arrays
    uint64_t* keys_in = nullptr;
    uint64_t* keys_out = nullptr;
    int32_t* vals_in = nullptr;
    int32_t* vals_out = nullptr;
    Ray* sorted = nullptr;
    TraceItem* src_items = nullptr;  // items with original rays, ray_begin = offset in sorted order
    float* bounds = nullptr;         // 6 floats per item
    void* cub_temp = nullptr;
    size_t cub_temp_bytes = 0;
    int end_bit = 64;
    int n_kernels = 0;  // kernels one sort_plan_run launches (counted from a captured graph)
};
rq_status sort_plan_create(const std::vector<TraceItem>& items, const std::vector<float>& bounds, SortPlan& plan);
rq_status sort_plan_run(SortPlan& plan, cudaStream_t s);
void sort_plan_destroy(SortPlan& plan);
int sort_plan_kernel_count(const SortPlan& plan);

}  // namespace rq
