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

// Which kernel a launch takes.  k_trace, a lane per ray, has the higher throughput; but a small launch lasts
// as long as its longest chain of node visits, and there k_trace_oct, eight lanes per ray, is faster.  Of
// asteroid-like bodies of 4 k / 40 k / 500 k triangles, times of k_trace to k_trace_oct, over the number of rays:
//   random closest-hit rays  2 k 1.44 / 1.53 / 1.46, 21 k 1.03 / 1.10 / 1.18, 31 k 0.89 / 0.95 / 1.08, 40 k 0.79 / 0.82 / 0.95
//   random any-hit rays      2 k 1.45 / 1.40 / 1.50, 21 k 1.15 / 1.19 / 1.20, 31 k 0.99 / 1.07 / 1.18, 40 k 0.85 / 0.95 / 1.02
//   path-traced images       21 k 1.08 / 1.28 / 1.39, 31 k 0.99 / 1.15 / 1.29, 58 k 0.89 / 1.04 / 1.20, 78 k 0.86 / 0.98 / 1.12
// (a buffer's coherent rays cross earlier: 21 k 0.94 / 0.86 / 0.93).  Jobs with FP64 work per ray stay with
// k_trace (OCT_NEVER): a warp's FP64 instruction takes the same 16 cycles for four rays as for 32.  So do
// scenes of fewer than SMALL_SCENE triangles, whose rays are done in a few nodes.
constexpr uint32_t OCT_ITEMS = 28000, OCT_ITEMS_MID = 40000, OCT_ITEMS_DEEP = 80000, OCT_DEEP_TRIS = 32768, SMALL_SCENE = 1024;
// A job's kOct: OCT_NEVER; OCT_DEEP (the default): up to OCT_ITEMS, in scenes of OCT_DEEP_TRIS triangles
// OCT_ITEMS_DEEP; OCT_MID: there up to OCT_ITEMS_MID; or OCT_COUNT: as OCT_DEEP, but the host knows only
// a bound far above the usual count, so both kernels are launched and the one that the count on the device
// does not call for returns at once.
enum { OCT_NEVER, OCT_MID, OCT_DEEP, OCT_COUNT };
template <class J, class = void>
struct trace_oct {
    static constexpr int value = OCT_DEEP;
};
template <class J>
struct trace_oct<J, std::void_t<decltype(J::kOct)>> {
    static constexpr int value = J::kOct;
};

// Jobs whose rays may be incoherent (kCoop) are traced with traverse_coop, unless the launch says that they
// are not (first shadow rays: 2048^2 of them 3 % slower with it) or the scene is of fewer than SMALL_SCENE
// triangles (a Cornell box's path-traced image: 563 us with it, 446 without; few specular rays of a served wave do
// not show it, srp_wave_stages_dev's caller in render.cu).  A job over a buffer of rays
// (JobBase) asks per warp (rays_apart).  Camera, beam and sun rays are coherent.
template <class J, class = void>
struct trace_coop {
    static constexpr bool value = false;
};
template <class J>
struct trace_coop<J, std::void_t<decltype(J::kCoop)>> {
    static constexpr bool value = J::kCoop;
};

// Jobs with many items that need no traversal (kGroups) name the groups of 32 items that a grab of a large
// launch takes: where most items end at once, the atomics on the one queue counter are the limit.
template <class J, class = void>
struct trace_groups {
    static constexpr bool value = false;
};
template <class J>
struct trace_groups<J, std::void_t<decltype(J::kGroups)>> {
    static constexpr bool value = J::kGroups;
};

// Persistent ray-queue kernel.  Each warp takes 32 consecutive items per atomic grab, or, with chunk > 1, a
// guided number of up to `chunk` times 32, shrinking with the work left so that the last grabs stay
// small (few atomics on the queue counter while much work is left, balance at the end).  queue: the next
// item, zero at the start.  A count of at most `over` items is left to the other kernel.  grab: chunk
// | groups << 8 (trace_groups) | GRAB_RESET: leave the queue at zero (queue[1] counts the blocks that have finished).
constexpr uint32_t GRAB_RESET = 1u << 31;

__device__ __forceinline__ void queue_reset(uint32_t* queue, uint32_t grab) {
    if (grab & GRAB_RESET) {   // the last block to finish leaves both counters zero for the next launch
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(queue + 1, 1u) == gridDim.x - 1u) queue[0] = queue[1] = 0u;
        }
    }
}

template <bool ANY, bool COUNT, bool COOP, class Job>
__global__ void __launch_bounds__(CRT_TRACE_BLOCK, trace_min_blocks<Job>::value) k_trace(SceneView sv, Job job, uint32_t n_items,
                                                            const uint32_t* __restrict__ n_dev,
                                                            uint32_t* __restrict__ queue, uint32_t* __restrict__ err,
                                                            unsigned long long* __restrict__ counters, uint32_t grab,
                                                            uint32_t over) {
    if (n_dev) n_items = *n_dev;   // item count produced by an earlier kernel on the stream
    if (n_items <= over) return;
    const int lane = threadIdx.x & 31;
    TravStats st{0u, 0u};
    uint32_t nrays = 0, nres = 0;
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
    const uint32_t chunk = grab & 0xFFu;
    while (true) {
        uint32_t base = 0, take = 1;
        if constexpr (trace_groups<Job>::value) take = grab >> 8 & 0xFFu;
        if (lane == 0) {
            if (chunk > 1) {
                const uint32_t cur = *reinterpret_cast<volatile uint32_t*>(queue);
                const uint32_t left = cur < n_items ? (n_items - cur) >> 5 : 0u;
                take = min(chunk, max(1u, left / (4u * warps_total)));
            }
            base = atomicAdd(queue, 32u * take);
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        take = __shfl_sync(0xffffffffu, take, 0);
        if (base >= n_items) break;
        for (const uint32_t end = base + 32u * take; base != end; base += 32u) {
            const uint32_t i = base + lane;
            TRay r;
            typename Job::Item it;
            const int kind = i < n_items ? (int)job.ray(i, r, it) : 0;
            if constexpr (COOP) {
                if (kind != 1) {
                    r.o = r.d = f3(0.f, 0.f, 1.f);
                    r.tmin = r.tmax = 0.f;
                }
                THit h;
                if constexpr (std::is_base_of_v<JobBase, Job>) {
                    if (rays_apart(sv, r, kind == 1)) h = traverse_coop<ANY, COUNT>(sv, r, kind == 1, trace_smem, st, err);
                    else if (kind == 1) h = traverse<ANY, COUNT>(sv, r, trace_smem, st, err);
                } else {
                    SceneView v{};
                    if (kind == 1) v = job.view(sv, it);
                    h = traverse_coop<ANY, COUNT>(v, r, kind == 1, trace_smem, st, err);
                }
                if (kind == 1) job.write(sv, i, r, h, it);
            } else if (kind == 1) {
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
    queue_reset(queue, grab);
}

// The ray queue with eight lanes per ray (traverse_oct): 1, 2 or 4 rays per warp and grab, the most that
// leave no warp without work.  A job's ray() runs on all of a ray's lanes (what it stores is the same
// from each), its write() on one.  A count above `upto` is left to k_trace.  6 blocks per SM (80
// registers): at 8 the kernels spill (a 128^2 render 92 -> 103 us).
template <bool ANY, bool COUNT, class Job>
__global__ void __launch_bounds__(CRT_TRACE_BLOCK, 6) k_trace_oct(SceneView sv, Job job, uint32_t n_items,
                                                                  const uint32_t* __restrict__ n_dev,
                                                                  uint32_t* __restrict__ queue,
                                                                  uint32_t* __restrict__ err,
                                                                  unsigned long long* __restrict__ counters,
                                                                  uint32_t grab, uint32_t upto) {
    if (n_dev) n_items = *n_dev;
    if (n_items > upto) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (CRT_TRACE_BLOCK / 32), per = n_items / warps;
    const uint32_t take = per >= 4u ? 4u : per >= 2u ? 2u : 1u;
    TravStats st{0u, 0u};
    uint32_t nrays = 0, nres = 0;
    while (true) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(queue, take);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n_items) break;
        const uint32_t i = base + (lane >> 3);
        TRay r;
        r.o = r.d = f3(0.f, 0.f, 1.f);
        r.tmin = r.tmax = 0.f;
        typename Job::Item it;
        const int kind = (lane >> 3) < take && i < n_items ? (int)job.ray(i, r, it) : 0;
        SceneView v{};
        if (kind == 1) v = job.view(sv, it);
        const THit h = traverse_oct<ANY, COUNT>(v, r, kind == 1, trace_smem, st, err);
        if (kind == 1 && (lane & 7u) == 0) job.write(sv, i, r, h, it);
        if (COUNT && (lane & 7u) == 0) {
            nrays += kind == 1;
            nres += kind == 2;
        }
    }
    if (COUNT) {
        atomicAdd(counters + 0, (unsigned long long)nrays);
        atomicAdd(counters + 1, (unsigned long long)st.nodes);
        atomicAdd(counters + 2, (unsigned long long)st.tris);
        atomicAdd(counters + 3, (unsigned long long)nres);
    }
    queue_reset(queue, grab);
}

// Resident blocks per SM of a kernel (a property of the kernel and its shared memory), asked for once.
template <class Kernel>
int resident_blocks(crt_context* ctx, Kernel* kernel, size_t smem, std::atomic<int>& known) {
    int blocks = known.load(std::memory_order_relaxed);
    if (!blocks) {
        blocks = occupancy_grid(ctx, (const void*)kernel, CRT_TRACE_BLOCK, smem) / ctx->sm_count;
        known.store(blocks, std::memory_order_relaxed);
    }
    return blocks;
}

// queue: a work counter that an earlier operation on the stream has zeroed; null: the context's own.
// There a small launch finds its counter at zero and leaves it so; past RESET_BLOCKS blocks the atomics of
// the finishing blocks take longer (2.4 us with 1216) than a memset before the launch, which overlaps
// the end of the work before it (256 rays: 23.0 us with the memset, 22.0 without).
constexpr int RESET_BLOCKS = 128;
inline uint32_t* own_queue(crt_context* ctx, uint32_t* q, int grid, uint32_t& grab) {
    if (q) return q;
    q = (uint32_t*)ctx_scratch(ctx, SCR_QUEUE, 256);
    if (grid <= RESET_BLOCKS) {
        grab |= GRAB_RESET;
        return q;
    }
    q += 8;   // words 0 and 1 stay zero for the small launches
    CRT_CUDA(cudaMemsetAsync(q, 0, sizeof(uint32_t), ctx->stream));
    return q;
}

template <bool ANY, bool COOP, class Job>
void launch_queue(crt_context* ctx, const SceneView& sv, const Job& job, uint32_t n_items, const uint32_t* n_dev,
                  uint32_t* q, uint32_t over) {
    static std::atomic<int> known[2] = {{0}, {0}};
    auto kernel = ctx->counting ? k_trace<ANY, true, COOP, Job> : k_trace<ANY, false, COOP, Job>;
    static_assert(!COOP || !trace_beam_bytes<Job>::value, "kept beams and the owners of dealt triangles share a place");
    constexpr size_t smem = (COOP ? COOP_SMEM : TRACE_SMEM) + trace_beam_bytes<Job>::value;
    int grid = resident_blocks(ctx, kernel, smem, known[ctx->counting]) * ctx->sm_count;
    const uint32_t need = (n_items + CRT_TRACE_BLOCK - 1) / CRT_TRACE_BLOCK;
    if ((uint32_t)grid > need) grid = (int)std::max<uint32_t>(need, 1u);
    uint32_t grab = ctx->queue_chunk ? ctx->queue_chunk : 1u;
    if constexpr (trace_groups<Job>::value)   // at least 16 grabs a warp
        grab |= std::max(1u, std::min(job.groups, (n_items >> 9) / (uint32_t)(grid * (CRT_TRACE_BLOCK / 32)))) << 8;
    q = own_queue(ctx, q, grid, grab);
    kernel<<<grid, CRT_TRACE_BLOCK, smem, ctx->stream>>>(sv, job, n_items, n_dev, q, ctx->d_error, ctx->d_counters, grab, over);
    check_launch(ctx, "k_trace");
}

// Launches a trace over n_items work items (or over *n_dev items when n_dev is given: n_items is then an
// upper bound).  tris: triangles of the smallest scene the rays meet, 0: keep to k_trace and traverse.
// coherent: neighbouring items' rays are alike (of a job that is otherwise taken not to be).
template <bool ANY, class Job>
void launch_trace(crt_context* ctx, const SceneView& sv, const Job& job, uint32_t n_items, const uint32_t* n_dev,
                  uint32_t* queue, size_t tris, bool coherent = false) {
    constexpr int oct = trace_oct<Job>::value;
    const bool counting = ctx->counting;
    uint32_t over = 0;
    if constexpr (oct != OCT_NEVER) {
        constexpr uint32_t deep = oct == OCT_MID ? OCT_ITEMS_MID : OCT_ITEMS_DEEP;
        const uint32_t limit = tris < SMALL_SCENE ? 0u : tris >= OCT_DEEP_TRIS ? deep : OCT_ITEMS;
        const bool fits = n_items <= limit, both = oct == OCT_COUNT && limit && !fits;
        if (fits || both) {
            static std::atomic<int> known[2] = {{0}, {0}};
            auto kernel = counting ? k_trace_oct<ANY, true, Job> : k_trace_oct<ANY, false, Job>;
            const uint32_t want = std::max<uint32_t>((std::min(n_items, limit) + CRT_TRACE_BLOCK / 32 - 1) / (CRT_TRACE_BLOCK / 32), 1u);
            const int grid = (int)std::min<uint32_t>((uint32_t)(resident_blocks(ctx, kernel, OCT_SMEM, known[counting]) * ctx->sm_count), want);
            uint32_t grab = 0;
            uint32_t* q = own_queue(ctx, queue, grid, grab);
            kernel<<<grid, CRT_TRACE_BLOCK, OCT_SMEM, ctx->stream>>>(sv, job, n_items, n_dev, q, ctx->d_error, ctx->d_counters,
                                                                   grab, both ? limit : 0xFFFFFFFFu);
            check_launch(ctx, "k_trace_oct");
            if (fits) return;
            over = limit;
        }
    }
    if constexpr (trace_coop<Job>::value) {
        if (!coherent && tris >= SMALL_SCENE) {
            launch_queue<ANY, true>(ctx, sv, job, n_items, n_dev, queue, over);
            return;
        }
    }
    launch_queue<ANY, false>(ctx, sv, job, n_items, n_dev, queue, over);
}

template <bool ANY, class Job>
void launch_trace(crt_scene* s, const Job& job, uint32_t n_items) {
    launch_trace<ANY>(s->ctx, scene_view(s), job, n_items, nullptr, nullptr, s->n_tris);
}
