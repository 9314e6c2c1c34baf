// Persistent trace-kernel template shared by every query, plus surface reconstruction helpers.
#pragma once

#include "common.cuh"
#include "traverse.cuh"

#include <atomic>
#include <type_traits>

// resident blocks per SM the trace kernel is compiled for (registers per thread: 65536 / (128 x 8) = 64).
#ifndef CRT_TRACE_MIN_BLOCKS
#define CRT_TRACE_MIN_BLOCKS 8
#endif

__host__ __device__ __forceinline__ SceneView scene_view(const crt_scene* s) {
    SceneView v;
    v.nodes = s->nodes;
    v.tris = s->tris;
    v.leaf_prim = s->leaf_prim;
    v.leaf_vn = s->leaf_vn;
    v.leaf_entity = s->leaf_entity;
    v.entities = s->entities;
    v.n_tris = (uint32_t)s->n_tris;
    return v;
}

// SimpleCamera::pixel_to_ray in FP32 from the FP64-derived basis: d = normalize(a + u b + v c).
__device__ __forceinline__ TRay camera_ray(const CamBasis& c, float u, float v) {
    TRay r;
    const float3 d = f3(fmaf(v, c.c[0], fmaf(u, c.b[0], c.a[0])), fmaf(v, c.c[1], fmaf(u, c.b[1], c.a[1])),
                        fmaf(v, c.c[2], fmaf(u, c.b[2], c.a[2])));
    r.d = normalize3(d);
    r.o = f3(c.o[0], c.o[1], c.o[2]);
    r.tmin = 0.f;
    r.tmax = 3.402823466e38f;
    return r;
}

struct SurfacePoint {
    float3 x;           // u p1 + v p2 + (1-u-v) p0  (passes.hpp:53)
    float3 flat_n;      // normalize(n), left-handed (inward) like the reference
    float3 shading_n;   // smooth ? normalize(u vn1 + v vn2 + w vn0) : flat_n  (passes.hpp:179)
    uint32_t entity;
    uint32_t id;
};

__device__ __forceinline__ SurfacePoint surface_point(const SceneView& sv, const THit& h) {
    SurfacePoint sp;
    const float4* tp = sv.tris + 3ull * h.slot;
    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
    const float3 p0 = f3(a.x, a.y, a.z), n = f3(c.y, c.z, c.w);
    // u p1 + v p2 + (1 - u - v) p0 = p0 + u (p1 - p0) + v (p2 - p0)
    sp.x = tri_point(a, b, c, h.u, h.v);
    sp.flat_n = normalize3(n);
    sp.entity = __ldg(sv.leaf_entity + h.slot);
    const EntityDev& E = sv.entities[sp.entity];
    sp.id = E.id;
    if (E.smooth && sv.leaf_vn) {
        const float4* vp = sv.leaf_vn + 3ull * h.slot;
        const float4 v0 = __ldg(vp), v1 = __ldg(vp + 1), v2 = __ldg(vp + 2);
        const float w = 1.0f - h.u - h.v;
        sp.shading_n = normalize3(f3(h.u * v1.x + h.v * v2.x + w * v0.x, h.u * v1.y + h.v * v2.y + w * v0.y,
                                     h.u * v1.z + h.v * v2.z + w * v0.z));
    } else {
        sp.shading_n = sp.flat_n;
    }
    return sp;
}

// Jobs: ray(i, r, item) builds the ray of work item i and returns 1 to trace it, 0 when the item has
// no ray (padding), or 2 when the ray is resolved without a traversal (a miss known from a bounding
// test; the job has nothing to store, and the counting build counts it among the resolved rays);
// bool results mean 1 / 0.  view(sv, item) names the scene to traverse (requests of one launch may
// use different resident scenes), and write(sv, i, r, hit, item) stores the result.  JobBase
// supplies the single-scene defaults.
struct JobBase {
    struct Item {};
    __device__ __forceinline__ const SceneView& view(const SceneView& sv, const Item&) const { return sv; }
};

// Resident blocks per SM for one job type: CRT_TRACE_MIN_BLOCKS unless the job names its own
// (kMinBlocks): jobs whose rays come with a scene of their own and a skipped triangle need more
// registers than 8 blocks leave and spill there (a 2048^2 render with its shadow rays at 8 blocks 1583
// us, at 7 1560 us).  launch_trace sizes the persistent grid from the occupancy the kernel gets.
template <class J, class = void>
struct trace_min_blocks {
    static constexpr int value = CRT_TRACE_MIN_BLOCKS;
};
template <class J>
struct trace_min_blocks<J, std::void_t<decltype(J::kMinBlocks)>> {
    static constexpr int value = J::kMinBlocks;
};

// Jobs that keep the FP64 direction of a beam from ray() to write() (kKeepsBeam) hold it in shared memory
// while the ray is traversed: worked out again after it, it was half of a beam scan's FP64, which took 16
// cycles per instruction and warp (1024^2 beams 197 -> 187 us).
extern __shared__ __align__(16) unsigned char trace_smem[];
constexpr uint32_t TRACE_BEAM = 24u * CRT_TRACE_BLOCK;   // bytes, after TRACE_SMEM
__device__ __forceinline__ void beam_keep(const double d[3]) {
    double* s = reinterpret_cast<double*>(trace_smem + TRACE_SMEM) + threadIdx.x;
    for (int k = 0; k < 3; ++k) s[k * CRT_TRACE_BLOCK] = d[k];
}
__device__ __forceinline__ void beam_kept(double d[3]) {
    const double* s = reinterpret_cast<const double*>(trace_smem + TRACE_SMEM) + threadIdx.x;
    for (int k = 0; k < 3; ++k) d[k] = s[k * CRT_TRACE_BLOCK];
}
template <class J, class = void>
struct trace_beam_bytes {
    static constexpr uint32_t value = 0;
};
template <class J>
struct trace_beam_bytes<J, std::void_t<decltype(J::kKeepsBeam)>> {
    static constexpr uint32_t value = TRACE_BEAM;
};

// How a job's launches choose the items per warp (group_size): by the bound on the item count known to the
// host, the default; by the count on the device (kGroups = GROUPS_DEVICE), for jobs whose bound is far
// above the usual count (specular continuations of a sun-ray grid; waves of a mixed batch that hold
// nothing but one small query; the job's full_groups() says where it has FP64 items); or always 32 (GROUPS_FULL), for jobs with FP64 work per item, which
// takes the same time for a warp with one active lane (a 229 x 128 beam scan: 34 us, in small groups 53).
// A group size from the device is a register of every thread, which cost 1.7 % of a 2048^2 render's
// traces, so it is not the default.
enum { GROUPS_HOST, GROUPS_DEVICE, GROUPS_FULL };
template <class J, class = void>
struct trace_groups {
    static constexpr int value = GROUPS_HOST;
};
template <class J>
struct trace_groups<J, std::void_t<decltype(J::kGroups)>> {
    static constexpr int value = J::kGroups;
};

// Items a warp takes at a time in a launch of n items on `warps` warps: 32, one per lane, unless that
// would leave more than half of the warps without work; then fewer, the other lanes idle.  A small
// launch lasts as long as its slowest warp, and a warp of 32 rays is slower than its slowest ray by
// every node and triangle that only other lanes visit.  256 rays on 20 k triangles 37 -> 21.5 us,
// a 128^2 render 167 -> 142 us, one 250^2 sun-ray grid with two bounces 181 -> 137 us.  (Groups that also
// shrink at the end of a large launch cost it 1 - 3 %: its last rays then take more issue slots.)
// Scenes of fewer than SMALL_SCENE triangles always get 32: their rays are done in a few nodes, and the
// work per ray outside the traversal, repeated per warp, is what they wait for (27 k camera paths in a
// box of 36 triangles: 64 us, in groups of 8 67 us).
constexpr size_t SMALL_SCENE = 1024;
__host__ __device__ __forceinline__ uint32_t group_size(uint32_t n, uint32_t warps) {
    const uint32_t per = n / warps;
    return per >= 16u ? 32u : per >= 8u ? 16u : per >= 4u ? 8u : per >= 2u ? 4u : per >= 1u ? 2u : 1u;
}

// Persistent ray-queue kernel.  Each warp takes one group of consecutive items per atomic grab, or,
// with chunk > 1 and full groups, a guided number of up to `chunk` groups, shrinking with the work left
// so that the last grabs stay small (few atomics on the queue counter while much work is left, balance
// at the end).  queue: the next item, zero at the start.  grab: group size (0: from the count, GROUPS_DEVICE) | chunk << 8
// | GRAB_RESET: leave the queue at zero (queue[1] counts the blocks that have finished).
constexpr uint32_t GRAB_RESET = 1u << 31;

template <bool ANY, bool COUNT, class Job>
__global__ void __launch_bounds__(CRT_TRACE_BLOCK, trace_min_blocks<Job>::value) k_trace(SceneView sv, Job job, uint32_t n_items,
                                                            const uint32_t* __restrict__ n_dev,
                                                            uint32_t* __restrict__ queue, uint32_t* __restrict__ err,
                                                            unsigned long long* __restrict__ counters, uint32_t grab) {
    if (n_dev) n_items = *n_dev;   // item count produced by an earlier kernel on the stream
    const uint32_t lane = threadIdx.x & 31u;
    TravStats st{0u, 0u};
    uint32_t nrays = 0, nres = 0;
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
    const uint32_t chunk = (grab >> 8) & 0xFFu;
    uint32_t group = grab & 0xFFu;
    if constexpr (trace_groups<Job>::value == GROUPS_DEVICE)
        if (!group) group = job.full_groups() ? 32u : group_size(n_items, warps_total);
    while (true) {
        uint32_t base = 0, take = group;
        if (lane == 0) {
            if (chunk > 1 && group == 32u) {
                const uint32_t cur = *reinterpret_cast<volatile uint32_t*>(queue);
                const uint32_t left = cur < n_items ? (n_items - cur) >> 5 : 0u;
                take = 32u * min(chunk, max(1u, left / (4u * warps_total)));
            }
            base = atomicAdd(queue, take);
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        take = __shfl_sync(0xffffffffu, take, 0);
        if (base >= n_items) break;
        for (const uint32_t end = base + ((take + 31u) & ~31u); base != end; base += 32u) {
            const uint32_t i = base + lane;
            TRay r;
            typename Job::Item it;
            const int kind = lane < group && i < n_items ? (int)job.ray(i, r, it) : 0;
            if (kind == 1) {
                const THit h = traverse<ANY, COUNT>(job.view(sv, it), r, trace_smem, st, err);
                job.write(sv, i, r, h, it);
            }
            if (COUNT) {
                nrays += kind == 1;
                nres += kind == 2;
            }
        }
    }
    if (COUNT) {
        unsigned long long a = nrays, b = st.nodes, c = st.tris, d = nres;
        for (int o = 16; o; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
            d += __shfl_xor_sync(0xffffffffu, d, o);
        }
        if (lane == 0) {
            atomicAdd(counters + 0, a);
            atomicAdd(counters + 1, b);
            atomicAdd(counters + 2, c);
            if (d) atomicAdd(counters + 3, d);
        }
    }
    if (grab & GRAB_RESET) {   // the last block to finish leaves both counters zero for the next launch
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(queue + 1, 1u) == gridDim.x - 1u) queue[0] = queue[1] = 0u;
        }
    }
}

// Launches the persistent trace kernel over n_items work items (or over *n_dev items when n_dev is
// given: n_items is then the upper bound used to size the grid).  full_groups: 32 items per warp whatever
// the count (launches with FP64 items among others).
// queue: a work counter that an earlier operation on the stream has zeroed; null: the context's own.
// There a small launch finds its counter at zero and leaves it so; past RESET_BLOCKS blocks the atomics of
// the finishing blocks take longer (2.4 us with 1216) than a memset before the launch, which overlaps
// the end of the work before it (256 rays: 23.0 us with the memset, 22.0 without).
constexpr int RESET_BLOCKS = 128;
template <bool ANY, class Job>
void launch_trace(crt_context* ctx, const SceneView& sv, const Job& job, uint32_t n_items,
                  const uint32_t* n_dev = nullptr, uint32_t* queue = nullptr, bool full_groups = false) {
    const size_t smem = TRACE_SMEM + trace_beam_bytes<Job>::value;
    static std::atomic<int> per_sm[2] = {{0}, {0}};   // resident blocks per SM, a property of the kernel
    int blocks = per_sm[ctx->counting].load(std::memory_order_relaxed);
    if (!blocks) {
        const void* kfn = ctx->counting ? (const void*)k_trace<ANY, true, Job> : (const void*)k_trace<ANY, false, Job>;
        blocks = occupancy_grid(ctx, kfn, CRT_TRACE_BLOCK, smem) / ctx->sm_count;
        per_sm[ctx->counting].store(blocks, std::memory_order_relaxed);
    }
    int grid = blocks * ctx->sm_count;
    constexpr int groups = trace_groups<Job>::value;
    full_groups = full_groups || groups == GROUPS_FULL || (sv.nodes && sv.n_tris < SMALL_SCENE);
    // at most one warp per group (per item where groups may be smaller than 32)
    const uint32_t per_block = full_groups ? CRT_TRACE_BLOCK : CRT_TRACE_BLOCK / 32;
    const uint32_t need = std::max<uint32_t>((n_items + per_block - 1) / per_block, 1u);
    if ((uint32_t)grid > need) grid = (int)need;
    const uint32_t group = full_groups ? 32u : groups == GROUPS_DEVICE ? 0u : group_size(n_items, (uint32_t)grid * (CRT_TRACE_BLOCK / 32));
    uint32_t grab = group | (ctx->queue_chunk ? ctx->queue_chunk : 1u) << 8;
    if (!queue) {
        queue = (uint32_t*)ctx_scratch(ctx, SCR_QUEUE, 256);
        if (grid <= RESET_BLOCKS) {
            grab |= GRAB_RESET;
        } else {
            queue += 8;   // words 0 and 1 stay zero for the small launches
            CRT_CUDA(cudaMemsetAsync(queue, 0, sizeof(uint32_t), ctx->stream));
        }
    }
    if (ctx->counting)
        k_trace<ANY, true, Job><<<grid, CRT_TRACE_BLOCK, smem, ctx->stream>>>(sv, job, n_items, n_dev, queue,
                                                                             ctx->d_error, ctx->d_counters, grab);
    else
        k_trace<ANY, false, Job><<<grid, CRT_TRACE_BLOCK, smem, ctx->stream>>>(sv, job, n_items, n_dev, queue,
                                                                              ctx->d_error, ctx->d_counters, grab);
    check_launch(ctx, "k_trace");
}

template <bool ANY, class Job>
void launch_trace(crt_scene* s, const Job& job, uint32_t n_items, const uint32_t* n_dev = nullptr,
                  uint32_t* queue = nullptr) {
    launch_trace<ANY>(s->ctx, scene_view(s), job, n_items, n_dev, queue);
}
