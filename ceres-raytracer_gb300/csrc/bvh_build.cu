// GPU BVH construction for a scene (replaces SweepSahBuilder + ParallelReinsertionOptimizer +
// NodeLayoutOptimizer of the reference, lib/bvh/sweep_sah_builder.hpp:43-111,
// parallel_reinsertion_optimizer.hpp:140-211, node_layout_optimizer.hpp:30-92).
//
// Pipeline, one stream; the host waits once for the SAH levels and once for the collapse levels (more
// only for trees much deeper than balanced ones):
//   k_transform      entity transform in FP64 (transform.hpp:43-85), FP32 triangle records
//                    (p0, p1, p2, n), exact FP32 boxes, centroids, normals
//   k_bounds         scene and centroid bounds (order-preserving integer atomics)
//   k_morton         30-bit Morton codes of centroids in the centroid bounds
//   radix_sort       stable LSD radix sort, 8-bit digits, 4 passes (histogram / scan / scatter)
//   sah_topology     binned-SAH tree over the Morton order (the default; else k_karras)
//   k_karras         binary radix tree (Karras, "Maximizing parallelism in the construction of
//                    BVHs, octrees, and k-d trees", HPG 2012); ties broken by index
//   k_refit          bottom-up boxes and collapse costs, second arrival at each node does the
//                    union
//   k_collapse       top-down, level-synchronous collapse into 8-wide nodes by a surface-area
//                    cost dynamic program over the binary tree (costs computed in the refit:
//                    each wide node spreads its 8 slots over subtrees where that is cheaper than
//                    keeping them whole); children with <= 3 triangles become leaves, slots ordered by octant, child boxes quantised to 8 bits
//                    (Ylitie, Karras, Laine, "Efficient incoherent ray traversal on GPUs through
//                    compressed wide BVHs", HPG 2017); leaf triangles written contiguously.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

namespace {

constexpr int BLOCK = 256;

struct EntXform {
    double scale;
    double pos[3];
    double rot[9];
    uint32_t first;      // first scene primitive of this entity
    uint32_t has_vn;
};

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 d3sub(D3 a, D3 b) { return {ds(a.x, b.x), ds(a.y, b.y), ds(a.z, b.z)}; }
__device__ __forceinline__ D3 d3add(D3 a, D3 b) { return {da(a.x, b.x), da(a.y, b.y), da(a.z, b.z)}; }
__device__ __forceinline__ D3 d3scl(D3 a, double s) { return {dm(a.x, s), dm(a.y, s), dm(a.z, s)}; }
// transform.hpp:22-28 rotate(): rows of R, left-to-right sums, no fused multiply-add
__device__ __forceinline__ D3 d3rot(D3 v, const double* R) {
    return {da(da(dm(R[0], v.x), dm(R[1], v.y)), dm(R[2], v.z)), da(da(dm(R[3], v.x), dm(R[4], v.y)), dm(R[5], v.z)),
            da(da(dm(R[6], v.x), dm(R[7], v.y)), dm(R[8], v.z))};
}
// bvh::cross (vector.hpp:161-169)
__device__ __forceinline__ D3 d3cross(D3 a, D3 b) {
    return {ds(dm(a.y, b.z), dm(a.z, b.y)), ds(dm(a.z, b.x), dm(a.x, b.z)), ds(dm(a.x, b.y), dm(a.y, b.x))};
}

// Order-preserving float <-> uint32 key for atomic min/max.
__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float fkey_inv(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}

// ---------------------------------------------------------------- K0 transform
__global__ void k_transform(const float* __restrict__ xyz, const float* __restrict__ vn, const EntXform* __restrict__ xf,
                            uint32_t n_ents, uint32_t n, float4* __restrict__ geo, float4* __restrict__ vn_out,
                            uint32_t* __restrict__ prim_ent, float4* __restrict__ box, float4* __restrict__ cen) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // entity of primitive i: last entity whose first <= i (few entities; linear search is fine)
    uint32_t e = 0;
    for (uint32_t k = 1; k < n_ents; ++k)
        if (xf[k].first <= i) e = k;
    const EntXform& X = xf[e];
    const float* q = xyz + 9ull * i;
    const D3 p0 = {q[0], q[1], q[2]}, p1 = {q[3], q[4], q[5]}, p2 = {q[6], q[7], q[8]};
    // resize_triangles, rotate_triangles, translate_triangles (p' = R (s p) + t), applied to each vertex
    // directly so that a vertex shared by several triangles gets one FP32 value in all of them (the
    // watertight test relies on it).  The reference carries each triangle as p0, e1 = p0 - p1,
    // e2 = p2 - p0 through the three steps (triangle.hpp:31-33, 81-82); the results differ by FP64
    // rounding only.
    const D3 t = {X.pos[0], X.pos[1], X.pos[2]};
    const D3 a = d3add(d3rot(d3scl(p0, X.scale), X.rot), t);
    const D3 b = d3add(d3rot(d3scl(p1, X.scale), X.rot), t);
    const D3 c = d3add(d3rot(d3scl(p2, X.scale), X.rot), t);
    const D3 nn = d3cross(d3sub(a, b), d3sub(c, a));   // n = e1 x e2
    const float P[3][3] = {{(float)a.x, (float)a.y, (float)a.z}, {(float)b.x, (float)b.y, (float)b.z},
                           {(float)c.x, (float)c.y, (float)c.z}};
    geo[3ull * i + 0] = make_float4(P[0][0], P[0][1], P[0][2], P[1][0]);
    geo[3ull * i + 1] = make_float4(P[1][1], P[1][2], P[2][0], P[2][1]);
    geo[3ull * i + 2] = make_float4(P[2][2], (float)nn.x, (float)nn.y, (float)nn.z);
    // box of the FP32 triangle (exact), centroid of its vertices
    float lo[3], hi[3], cc[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = fminf(P[0][k], fminf(P[1][k], P[2][k]));
        hi[k] = fmaxf(P[0][k], fmaxf(P[1][k], P[2][k]));
        cc[k] = (float)(((double)P[0][k] + (double)P[1][k] + (double)P[2][k]) * (1.0 / 3.0));
    }
    box[2ull * i] = make_float4(lo[0], lo[1], lo[2], 0.f);
    box[2ull * i + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    cen[i] = make_float4(cc[0], cc[1], cc[2], 0.f);
    prim_ent[i] = e;
    if (vn_out) {
        if (X.has_vn && vn) {
            const float* w = vn + 9ull * i;
            for (int k = 0; k < 3; ++k) {
                D3 v = d3rot(D3{w[3 * k], w[3 * k + 1], w[3 * k + 2]}, X.rot);
                vn_out[3ull * i + k] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
            }
        } else {
            for (int k = 0; k < 3; ++k) vn_out[3ull * i + k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// ---------------------------------------------------------------- K1 bounds
// keys[0..5] = scene box min xyz (as fkey, atomicMin) / max xyz (atomicMax); keys[6..11] centroid box
__global__ void k_bounds(const float4* __restrict__ box, const float4* __restrict__ cen, uint32_t n,
                         uint32_t* __restrict__ keys) {
    __shared__ uint32_t s[12];
    if (threadIdx.x < 12) s[threadIdx.x] = (threadIdx.x % 6) < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
    uint32_t lo[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
    uint32_t hi[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 a = box[2ull * i], b = box[2ull * i + 1], c = cen[i];
        float av[3] = {a.x, a.y, a.z}, bv[3] = {b.x, b.y, b.z}, cv[3] = {c.x, c.y, c.z};
        for (int k = 0; k < 3; ++k) {
            lo[k] = min(lo[k], fkey(av[k]));
            hi[k] = max(hi[k], fkey(bv[k]));
            lo[3 + k] = min(lo[3 + k], fkey(cv[k]));
            hi[3 + k] = max(hi[3 + k], fkey(cv[k]));
        }
    }
    for (int k = 0; k < 6; ++k) {
        for (int o = 16; o; o >>= 1) {
            lo[k] = min(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = max(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int k = 0; k < 3; ++k) {
            atomicMin(&s[k], lo[k]);
            atomicMax(&s[3 + k], hi[k]);
            atomicMin(&s[6 + k], lo[3 + k]);
            atomicMax(&s[9 + k], hi[3 + k]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        if ((threadIdx.x % 6) < 3) atomicMin(&keys[threadIdx.x], s[threadIdx.x]);
        else atomicMax(&keys[threadIdx.x], s[threadIdx.x]);
    }
}

// ---------------------------------------------------------------- K2 Morton codes
__device__ __forceinline__ uint32_t expand10(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}
__global__ void k_morton(const float4* __restrict__ cen, uint32_t n, const uint32_t* __restrict__ keys,
                         uint32_t* __restrict__ code, uint32_t* __restrict__ idx) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float lo[3], ext[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = fkey_inv(keys[6 + k]);
        float h = fkey_inv(keys[9 + k]);
        ext[k] = h - lo[k];
    }
    float4 c = cen[i];
    float cv[3] = {c.x, c.y, c.z};
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
        float t = ext[k] > 0.f ? (cv[k] - lo[k]) / ext[k] : 0.5f;
        q[k] = (uint32_t)fminf(fmaxf(t * 1024.0f, 0.0f), 1023.0f);
    }
    code[i] = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
    idx[i] = i;
}

// ---------------------------------------------------------------- K3 stable LSD radix sort
constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;

__global__ void __launch_bounds__(SORT_THREADS) k_radix_hist(const uint32_t* __restrict__ keys, uint32_t n,
                                                               int shift, uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * SORT_TILE;
    for (int r = 0; r < SORT_ITEMS; ++r) {
        uint32_t i = base + r * SORT_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(keys[i] >> shift) & 0xFF], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// exclusive scan of m values with one block of 1024 threads, 8 consecutive values per thread at a time
// (one thread per contiguous part of the array took 25 us for 31 k values, this takes 8)
__global__ void __launch_bounds__(1024) k_scan(uint32_t* __restrict__ a, uint32_t m) {
    __shared__ uint32_t part[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < m; base += 8192u) {
        const uint32_t b = base + threadIdx.x * 8u;
        uint32_t v[8], s = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            v[k] = b + k < m ? a[b + k] : 0u;
            s += v[k];
        }
        uint32_t x = s;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[warp] = x;
        __syncthreads();
        uint32_t w = part[lane];   // every warp scans the 32 warp totals
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        const uint32_t before = warp ? __shfl_sync(0xFFFFFFFFu, w, warp - 1) : 0u;
        uint32_t run = carry + before + x - s;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (b + k < m) a[b + k] = run;
            run += v[k];
        }
        carry += __shfl_sync(0xFFFFFFFFu, w, 31);
        __syncthreads();   // `part` is rewritten by the next round
    }
}

// Stable scatter: items of a tile are ranked in tile order (round, warp, lane); within a warp,
// equal digits are ranked with __match_any_sync, across warps with per-round digit counts.
__global__ void __launch_bounds__(SORT_THREADS) k_radix_scatter(const uint32_t* __restrict__ kin,
                                                                  const uint32_t* __restrict__ vin,
                                                                  uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                                  uint32_t n, int shift,
                                                                  const uint32_t* __restrict__ offs) {
    constexpr int WARPS = SORT_THREADS / 32;
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[WARPS][256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    base[tid] = offs[tid * gridDim.x + blockIdx.x];
    const uint32_t tile = blockIdx.x * SORT_TILE;
    const uint32_t lt = (1u << lane) - 1u;
    for (int r = 0; r < SORT_ITEMS; ++r) {
        for (int w = 0; w < WARPS; ++w) wcnt[w][tid] = 0;
        __syncthreads();
        const uint32_t i = tile + r * SORT_THREADS + tid;
        const bool valid = i < n;
        uint32_t k = 0, v = 0, d = 256 + lane;
        if (valid) {
            k = kin[i];
            v = vin[i];
            d = (k >> shift) & 0xFF;
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rank = __popc(peers & lt);
        if (valid && rank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t pos = base[d] + rank;
            for (int w = 0; w < warp; ++w) pos += wcnt[w][d];
            kout[pos] = k;
            vout[pos] = v;
        }
        __syncthreads();
        uint32_t add = 0;
        for (int w = 0; w < WARPS; ++w) add += wcnt[w][tid];
        base[tid] += add;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- K4 Karras radix tree
__device__ __forceinline__ int delta(const uint32_t* __restrict__ code, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = code[i], b = code[j];
    if (a == b) return 32 + __clz((uint32_t)(i ^ j));
    return __clz(a ^ b);
}
// children: >= 0 internal index, < 0 leaf ~j (sorted position j)
__global__ void k_karras(const uint32_t* __restrict__ code, int n, int2* __restrict__ child, int2* __restrict__ range,
                         int* __restrict__ parent) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(code, n, i, i + 1) - delta(code, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(code, n, i, i - d);
    int lmax = 2;
    while (delta(code, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(code, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(code, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(code, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = (lo == gamma) ? ~gamma : gamma;
    const int right = (hi == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    child[i] = make_int2(left, right);
    range[i] = make_int2(lo, hi);
    parent[left >= 0 ? left : (n - 1) + ~left] = i;
    parent[right >= 0 ? right : (n - 1) + ~right] = i;
}

// ---------------------------------------------------------------- refit + collapse costs
// Surface-area costs for the 8-wide collapse (a dynamic program over the binary tree): for an
// internal node b, dp[8 b] = cost of b as one root of a wide node's slot (a leaf when it holds at
// most 3 triangles, else an 8-wide node: COST_NODE area + the best spread of 8 slots over its
// children), dp[8 b + j - 1] = cost of spreading j = 2..8 slots over its two children.  The ratio
// triangle-test cost `cost_tri` is relative to an 8-wide node test (COST_NODE = 1): the default
// 0.15 is the trace kernel's instruction ratio (~40 : ~280), best for coherent rays; incoherent
// multi-bounce workloads prefer smaller leaves (a larger cost, crt_tuning.collapse_tri_cost).
constexpr float COST_NODE = 1.0f;

__device__ __forceinline__ float box_area(const float4& lo, const float4& hi) {
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// cost of child `ref` given i slots (1..8): out[i]
__device__ __forceinline__ void dp_child(const float* __restrict__ dp, int ref, float leaf_area, float cost_tri,
                                         float out[9]) {
    if (ref < 0) {
        const float v = cost_tri * leaf_area;
        for (int i = 1; i <= 8; ++i) out[i] = v;
        return;
    }
    const float4* d = reinterpret_cast<const float4*>(dp + 8ull * ref);
    const float4 a = __ldcg(d), b = __ldcg(d + 1);
    out[1] = a.x;
    out[2] = fminf(a.x, a.y);
    out[3] = fminf(a.x, a.z);
    out[4] = fminf(a.x, a.w);
    out[5] = fminf(a.x, b.x);
    out[6] = fminf(a.x, b.y);
    out[7] = fminf(a.x, b.z);
    out[8] = fminf(a.x, b.w);
}

// node boxes: 2 float4 per node; internal nodes [0, n-1), leaves [n-1, 2n-1)
__global__ void k_refit(const uint32_t* __restrict__ sorted, const float4* __restrict__ tbox, int n,
                        const int2* __restrict__ child, const int* __restrict__ parent, float4* nbox,
                        uint32_t* __restrict__ flags, const int2* __restrict__ range, float* __restrict__ dp,
                        float cost_tri, uint32_t* __restrict__ err) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t p = sorted[j];
    float4 lo = tbox[2ull * p], hi = tbox[2ull * p + 1];
    nbox[2ull * (n - 1 + j)] = lo;
    nbox[2ull * (n - 1 + j) + 1] = hi;
    int node = parent[n - 1 + j];
    for (int steps = 0; node >= 0; ++steps) {
        if (steps >= 1024) {   // deeper than any tree built here, or damaged links: report, do not loop
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
            return;
        }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0) return;   // first arrival: the sibling finishes the union
        const int2 c = child[node];
        const size_t a = c.x >= 0 ? (size_t)c.x : (size_t)(n - 1 + ~c.x);
        const size_t b = c.y >= 0 ? (size_t)c.y : (size_t)(n - 1 + ~c.y);
        const float4 alo = __ldcg(&nbox[2 * a]), ahi = __ldcg(&nbox[2 * a + 1]);
        const float4 blo = __ldcg(&nbox[2 * b]), bhi = __ldcg(&nbox[2 * b + 1]);
        lo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), 0.f);
        hi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.f);
        __stcg(&nbox[2ull * node], lo);
        __stcg(&nbox[2ull * node + 1], hi);
        if (dp) {
            float cl[9], cr[9];
            dp_child(dp, c.x, box_area(alo, ahi), cost_tri, cl);
            dp_child(dp, c.y, box_area(blo, bhi), cost_tri, cr);
            float* out = dp + 8ull * node;
            float dist8 = 3.0e38f;
            for (int j = 2; j <= 8; ++j) {
                float best = 3.0e38f;
                for (int k = 1; k < j; ++k) best = fminf(best, cl[k] + cr[j - k]);
                __stcg(out + j - 1, best);
                dist8 = best;
            }
            const int2 r = range[node];
            const float a = box_area(lo, hi);
            const float c_int = COST_NODE * a + dist8;
            const float c_leaf = r.y - r.x + 1 <= 3 ? cost_tri * (float)(r.y - r.x + 1) * a : 3.0e38f;
            __stcg(out, fminf(c_int, c_leaf));
        }
        node = parent[node];
    }
}

// ---------------------------------------------------------------- treelet restructuring
// Tree optimisation after the topology build, in place of the reference's parallel reinsertion
// (ParallelReinsertionOptimizer::optimize, parallel_reinsertion_optimizer.hpp:140-211): treelet
// restructuring after Karras and Aila, "Fast parallel construction of high-quality bounding volume
// hierarchies" (HPG 2013).  A treelet is a node R with up to TL_LEAVES descendants as leaves, grown
// from R's two children by repeatedly opening the leaf of largest surface area; its internal nodes
// are rebuilt into the topology of least summed surface area (the surface-area cost with the leaf
// subtrees fixed: their costs are the same in every topology), found by a dynamic program over the
// 2^7 - 1 subsets of leaves, one warp per treelet.  Node indices, boxes of R and everything outside
// the treelet stay; only child / parent links of its internal nodes and their boxes change.
// Treelets of one launch must not share nodes: a launch takes the roots whose depth is = r (mod 7),
// and a treelet from depth d holds internal nodes at depths d .. d + 5 and leaves at depths up to
// d + 6, so two roots 7 or more levels apart, or in disjoint subtrees, touch disjoint nodes.  Depths
// are recomputed before every launch.  Afterwards k_tl_count / k_tl_position / k_tl_relayout renumber
// the leaves in depth-first order, so every subtree is again a contiguous range of sorted positions
// (what the refit and the 8-wide collapse read).
constexpr int TL_LEAVES = 7;
constexpr int TL_WARPS = 4;

__device__ __forceinline__ size_t tl_index(int n, int ref) { return ref >= 0 ? (size_t)ref : (size_t)(n - 1 + ~ref); }

// Treelet roots of one launch: the internal nodes whose depth (root 0, found by walking up the parent
// links) is = cls (mod 7) and that hold at least three leaves, listed in any order (treelets of a launch
// are independent).
__global__ void k_tl_roots(const int* __restrict__ parent, const int2* __restrict__ child, int n, int cls,
                           int* __restrict__ list, uint32_t* __restrict__ count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool root = false;
    if (i < n - 1) {
        int d = 0, node = i;
        while (true) {
            const int p = parent[node];
            if (p < 0 || d >= 255) break;
            node = p;
            ++d;
        }
        const int2 c = child[i];
        root = d < 255 && d % 7 == cls && (c.x >= 0 || c.y >= 0);   // 255: deeper than tracked
    }
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, root);
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (root) list[base + __popc(m & ((1u << lane) - 1u))] = i;
}

// The subsets of 7 leaves by size (ascending within a size), sizes 2 .. 5, and where each size begins.
__constant__ uint8_t TL_SUBSETS[112] = {
    3,  5,  6,  9,  10, 12, 17, 18, 20, 24, 33, 34, 36, 40, 48, 65, 66, 68, 72, 80, 96,   // 2
    7,  11, 13, 14, 19, 21, 22, 25, 26, 28, 35, 37, 38, 41, 42, 44, 49, 50, 52, 56, 67, 69, 70, 73, 74, 76, 81, 82,
    84, 88, 97, 98, 100, 104, 112,   // 3
    15, 23, 27, 29, 30, 39, 43, 45, 46, 51, 53, 54, 57, 58, 60, 71, 75, 77, 78, 83, 85, 86, 89, 90, 92, 99, 101, 102,
    105, 106, 108, 113, 114, 116, 120,   // 4
    31, 47, 55, 59, 61, 62, 79, 87, 91, 93, 94, 103, 107, 109, 110, 115, 117, 118, 121, 122, 124};   // 5

// keeps the cheaper partition; of equal ones the larger subset
__device__ __forceinline__ void tl_better(float& best, uint32_t& bp, float c, uint32_t P) {
    if (c < best || (c == best && P > bp)) {
        best = c;
        bp = P;
    }
}

// One warp per treelet.  What bounds it: the chain of dependent loads that grows the treelet (each
// opened node gives the next two boxes) and the dynamic program's 966 partitions, both of which one
// lane walked before; now the leaves sit in lanes, and the partitions of a size are spread over lanes
// (one lane a subset up to size 5, four lanes a subset of 6, all lanes for 7).  500 k triangles, seven
// launches: 2516 -> 632 us.
__global__ void __launch_bounds__(32 * TL_WARPS) k_treelet(int2* __restrict__ child, int* __restrict__ parent,
                                                          float4* __restrict__ nbox, const int* __restrict__ list,
                                                          const uint32_t* __restrict__ count, int n) {
    __shared__ float s_area[TL_WARPS][128];
    __shared__ float s_cost[TL_WARPS][128];
    __shared__ uint8_t s_part[TL_WARPS][128];
    __shared__ float s_box[TL_WARPS][TL_LEAVES][6];
    __shared__ int s_leaf[TL_WARPS][TL_LEAVES];
    __shared__ int s_int[TL_WARPS][TL_LEAVES - 1];
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t warps = gridDim.x * TL_WARPS, todo = *count;
    for (uint32_t item = blockIdx.x * TL_WARPS + w; item < todo; item += warps) {
        const int R = list[item];
        // grow the treelet: open the leaf of largest area that is an internal node (of equal ones the
        // first); lane k holds leaf k
        const int2 c = child[R];
        int ref = lane == 0 ? c.x : c.y, nl = 2;
        float4 lo, hi;
        uint32_t key = 0;   // area of an internal leaf as an ordered integer, 0: none
        auto load = [&]() {
            const size_t bi = tl_index(n, ref);
            lo = nbox[2 * bi];
            hi = nbox[2 * bi + 1];
            key = ref >= 0 ? __float_as_uint(box_area(lo, hi)) + 1u : 0u;
        };
        if (lane < 2) load();
        float old = box_area(nbox[2 * (size_t)R], nbox[2 * (size_t)R + 1]);
        if (lane == 0) s_int[w][0] = R;
        while (nl < TL_LEAVES) {
            const uint32_t top = __reduce_max_sync(ALL, key);
            if (!top) break;
            const int best = __ffs(__ballot_sync(ALL, key == top)) - 1;
            const int L = __shfl_sync(ALL, ref, best);
            old += __uint_as_float(top - 1u);
            const int2 cc = child[L];
            if (lane == 0) s_int[w][nl - 1] = L;
            if (lane == best || lane == nl) {
                ref = lane == best ? cc.x : cc.y;
                load();
            }
            ++nl;
        }
        if (nl < 3) continue;   // uniform: two triangles
        if (lane < nl) {
            s_leaf[w][lane] = ref;
            s_box[w][lane][0] = lo.x; s_box[w][lane][1] = lo.y; s_box[w][lane][2] = lo.z;
            s_box[w][lane][3] = hi.x; s_box[w][lane][4] = hi.y; s_box[w][lane][5] = hi.z;
        }
        __syncwarp();
        const uint32_t full = (1u << nl) - 1u;
        {   // surface area of the union of each subset's boxes: lane takes subsets lane, lane + 32, ...
            float ulo[4][3], uhi[4][3];
            for (int q = 0; q < 4; ++q)
                for (int a = 0; a < 3; ++a) {
                    ulo[q][a] = 3.0e38f;
                    uhi[q][a] = -3.0e38f;
                }
            for (int k = 0; k < nl; ++k) {
                const float b0 = s_box[w][k][0], b1 = s_box[w][k][1], b2 = s_box[w][k][2];
                const float b3 = s_box[w][k][3], b4 = s_box[w][k][4], b5 = s_box[w][k][5];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (((uint32_t)(lane + 32 * q) >> k) & 1u) {
                        ulo[q][0] = fminf(ulo[q][0], b0); ulo[q][1] = fminf(ulo[q][1], b1); ulo[q][2] = fminf(ulo[q][2], b2);
                        uhi[q][0] = fmaxf(uhi[q][0], b3); uhi[q][1] = fmaxf(uhi[q][1], b4); uhi[q][2] = fmaxf(uhi[q][2], b5);
                    }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float dx = uhi[q][0] - ulo[q][0], dy = uhi[q][1] - ulo[q][1], dz = uhi[q][2] - ulo[q][2];
                s_area[w][lane + 32 * q] = dx * dy + dy * dz + dz * dx;
                s_cost[w][lane + 32 * q] = 0.f;
            }
        }
        __syncwarp();
        // cost of the best subtree over each subset, by subset size.  A partition is (P, S ^ P) with P
        // holding the lowest leaf of S.
        const float* cost = s_cost[w];
        constexpr int begin[4] = {0, 21, 56, 91}, end[4] = {21, 56, 91, 112};
#pragma unroll 1
        for (int size = 2; size <= min(nl, 5); ++size) {
            for (int t = begin[size - 2] + lane; t < end[size - 2]; t += 32) {
                const uint32_t S = TL_SUBSETS[t];
                if (S > full) continue;
                const uint32_t low = S & (0u - S), rest = S ^ low;
                float best = 3.0e38f;
                uint32_t bp = low;
                for (uint32_t Q = rest; Q;) {
                    Q = (Q - 1) & rest;
                    const float v = cost[Q | low] + cost[rest ^ Q];
                    if (v < best) {
                        best = v;
                        bp = Q | low;
                    }
                }
                s_cost[w][S] = s_area[w][S] + best;
                s_part[w][S] = (uint8_t)bp;
            }
            __syncwarp();
        }
        if (nl >= 6) {   // subsets of 6: all leaves but leaf m; four lanes each
            const uint32_t m = (uint32_t)lane >> 2, S = 127u ^ (1u << m);
            const bool on = lane < 28 && S <= full;
            float best = 3.0e38f;
            uint32_t bp = S & (0u - S);
            if (on) {
                const uint32_t low = bp, rest = S ^ low;
                const int sh = m == 0 ? 2 : 1;
                for (uint32_t j = lane & 3; j < 31u; j += 4) {   // the j-th proper subset of rest
                    uint32_t Q = j << sh;
                    if (m > 0) Q = (Q & ((1u << m) - 1u)) | ((Q >> m) << (m + 1));
                    tl_better(best, bp, cost[Q | low] + cost[rest ^ Q], Q | low);
                }
            }
            for (int o = 1; o < 4; o <<= 1) tl_better(best, bp, __shfl_xor_sync(ALL, best, o), __shfl_xor_sync(ALL, bp, o));
            __syncwarp();
            if (on && (lane & 3) == 0) {
                s_cost[w][S] = s_area[w][S] + best;
                s_part[w][S] = (uint8_t)bp;
            }
            __syncwarp();
        }
        if (nl == 7) {   // all leaves: 63 partitions over the warp
            float best = 3.0e38f;
            uint32_t bp = 1u;
            for (uint32_t j = lane; j < 63u; j += 32) {
                const uint32_t Q = j << 1;
                tl_better(best, bp, cost[Q | 1u] + cost[126u ^ Q], Q | 1u);
            }
            for (int o = 1; o < 32; o <<= 1) tl_better(best, bp, __shfl_xor_sync(ALL, best, o), __shfl_xor_sync(ALL, bp, o));
            if (lane == 0) {
                s_cost[w][127] = s_area[w][127] + best;
                s_part[w][127] = (uint8_t)bp;
            }
            __syncwarp();
        }
        if (lane == 0 && s_cost[w][full] < old * (1.0f - 1e-5f)) {
            // rebuild: internal nodes reuse the treelet's indices (R stays the root)
            uint32_t stk_s[TL_LEAVES], ord_s[TL_LEAVES];
            int stk_n[TL_LEAVES], ord_n[TL_LEAVES];
            int sp = 0, no = 0, next = 1;
            stk_s[sp] = full;
            stk_n[sp++] = R;
            while (sp) {
                --sp;
                const uint32_t S = stk_s[sp];
                const int node = stk_n[sp];
                ord_s[no] = S;
                ord_n[no++] = node;
                const uint32_t P = s_part[w][S], Q = S ^ P;
                int ch[2];
                const uint32_t part[2] = {P, Q};
                for (int k = 0; k < 2; ++k) {
                    if (__popc(part[k]) == 1) {
                        ch[k] = s_leaf[w][__ffs(part[k]) - 1];
                    } else {
                        ch[k] = s_int[w][next++];
                        stk_s[sp] = part[k];
                        stk_n[sp++] = ch[k];
                    }
                    parent[tl_index(n, ch[k])] = node;
                }
                child[node] = make_int2(ch[0], ch[1]);
            }
            // boxes of the rebuilt internal nodes (R's box is unchanged)
            for (int k = 1; k < no; ++k) {
                float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
                for (int j = 0; j < nl; ++j)
                    if ((ord_s[k] >> j) & 1u)
                        for (int a = 0; a < 3; ++a) {
                            lo[a] = fminf(lo[a], s_box[w][j][a]);
                            hi[a] = fmaxf(hi[a], s_box[w][j][3 + a]);
                        }
                nbox[2 * (size_t)ord_n[k]] = make_float4(lo[0], lo[1], lo[2], 0.f);
                nbox[2 * (size_t)ord_n[k] + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
            }
        }
        __syncwarp();
    }
}

// boxes only (the treelet pass reads node areas): second arrival at each node does the union
// Every walk up the parent links below stops after TL_MAX_WALK steps with DEVERR_BUILD_OVERFLOW (a
// binary tree this deep, or a damaged one, is reported instead of looping).
constexpr int TL_MAX_WALK = 1024;

__global__ void k_tl_boxes(const uint32_t* __restrict__ sorted, const float4* __restrict__ tbox, int n,
                           const int2* __restrict__ child, const int* __restrict__ parent, float4* nbox,
                           uint32_t* __restrict__ flags, uint32_t* __restrict__ err) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t p = sorted[j];
    nbox[2ull * (n - 1 + j)] = tbox[2ull * p];
    nbox[2ull * (n - 1 + j) + 1] = tbox[2ull * p + 1];
    int node = parent[n - 1 + j];
    for (int steps = 0; node >= 0; ++steps) {
        if (steps >= TL_MAX_WALK) {
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
            return;
        }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0) return;
        const int2 c = child[node];
        const size_t a = tl_index(n, c.x), b = tl_index(n, c.y);
        const float4 alo = __ldcg(&nbox[2 * a]), ahi = __ldcg(&nbox[2 * a + 1]);
        const float4 blo = __ldcg(&nbox[2 * b]), bhi = __ldcg(&nbox[2 * b + 1]);
        __stcg(&nbox[2ull * node], make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), 0.f));
        __stcg(&nbox[2ull * node + 1], make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.f));
        node = parent[node];
    }
}

// triangles under every internal node: second arrival at each node adds its children's counts
__global__ void k_tl_count(int n, const int2* __restrict__ child, const int* __restrict__ parent,
                           int* __restrict__ cnt, uint32_t* __restrict__ flags, uint32_t* __restrict__ err) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    int node = parent[n - 1 + j];
    for (int steps = 0; node >= 0; ++steps) {
        if (steps >= TL_MAX_WALK) {
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
            return;
        }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0) return;
        const int2 c = child[node];
        const int a = c.x >= 0 ? __ldcg(&cnt[c.x]) : 1, b = c.y >= 0 ? __ldcg(&cnt[c.y]) : 1;
        __stcg(&cnt[node], a + b);
        node = parent[node];
    }
}

// depth-first position of every node (internal: of its first leaf): the triangles of the left
// siblings along the path to the root
__global__ void k_tl_position(int n, const int2* __restrict__ child, const int* __restrict__ parent,
                              const int* __restrict__ cnt, int* __restrict__ pos, uint32_t* __restrict__ err) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= 2 * n - 1) return;
    int node = x, p = 0;
    int ref = x < n - 1 ? x : ~(x - (n - 1));
    for (int steps = 0;; ++steps) {
        const int par = parent[node];
        if (par < 0) break;
        if (steps >= TL_MAX_WALK) {
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
            p = 0;
            break;
        }
        const int2 c = child[par];
        if (c.y == ref) p += c.x >= 0 ? cnt[c.x] : 1;
        node = par;
        ref = par;
    }
    pos[x] = p;
}

// renumber leaves by their depth-first position: sorted order, leaf references, leaf parents, ranges
__global__ void k_tl_relayout(int n, const int* __restrict__ pos, const int* __restrict__ cnt,
                              const uint32_t* __restrict__ sorted_in, uint32_t* __restrict__ sorted_out,
                              int2* __restrict__ child, int2* __restrict__ range, const int* __restrict__ parent_in,
                              int* __restrict__ leaf_parent_out, uint32_t* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {   // leaf at sorted position i moves to pos[n - 1 + i]
        const int q = pos[n - 1 + i];
        if (q < 0 || q >= n) {
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
        } else {
            sorted_out[q] = sorted_in[i];
            leaf_parent_out[q] = parent_in[n - 1 + i];
        }
    }
    if (i < n - 1) {
        int2 c = child[i];
        const bool ok = (c.x >= 0 ? c.x < n - 1 : ~c.x < n) && (c.y >= 0 ? c.y < n - 1 : ~c.y < n) && cnt[i] >= 2 &&
                        pos[i] >= 0 && pos[i] + cnt[i] <= n;
        if (!ok) {
            atomicOr(err, (uint32_t)DEVERR_BUILD_OVERFLOW);
            return;
        }
        if (c.x < 0) c.x = ~pos[n - 1 + ~c.x];
        if (c.y < 0) c.y = ~pos[n - 1 + ~c.y];
        child[i] = c;
        range[i] = make_int2(pos[i], pos[i] + cnt[i] - 1);
    }
}

// ---------------------------------------------------------------- K5 collapse to 8-wide nodes
struct CollapseArgs {
    int n;                        // triangles
    const int2* child;            // binary children
    const int2* range;            // binary ranges
    const float4* nbox;           // binary node boxes
    const uint32_t* sorted;       // sorted position -> scene primitive
    const float4* geo;            // triangle records, scene order
    const float4* vn;             // vertex normals, scene order (may be null)
    const uint32_t* prim_ent;     // entity per scene primitive
    WideNode* nodes;
    float4* tris;                 // leaf-order triangle records
    uint32_t* leaf_prim;
    float4* leaf_vn;
    uint32_t* leaf_entity;
    uint32_t* counters;           // [0] wide nodes used, [1] triangles placed
    uint32_t node_cap;
    uint32_t* err;
    const float* dp;              // collapse costs from k_refit
    float cost_tri;               // triangle-test cost relative to a node test
};

__device__ __forceinline__ size_t box_index(int n, int ref) { return ref >= 0 ? (size_t)ref : (size_t)(n - 1 + ~ref); }

// Quantisation grid of a node along one axis: p = lo - 2 q, q = 2^e with (hi - lo) / q <= 250 and q >= 4
// ulps of the largest coordinate; every child box is widened by one quantum on each side, so the decoded
// FP32 planes enclose the FP32 triangles with a margin of at least 4 ulps.
__device__ __forceinline__ void node_grid(float lo, float hi, float& p, int& ex) {
    const double ext = ((double)hi - (double)lo) / 250.0;
    int e = -126;
    if (ext > 0) {   // the least e with 2^e >= ext
        const double f = frexp(ext, &e);   // ext = f 2^e, f in [0.5, 1)
        if (f == 0.5) --e;
    }
    const float m = fmaxf(fabsf(lo), fabsf(hi));
    int em = -126;
    if (m > 0.f) {
        int fe;
        frexpf(m, &fe);          // m in [2^(fe-1), 2^fe)
        em = fe - 1 - 23 + 2;    // 4 ulps
    }
    ex = min(max(max(e, em), -126), 127);
    p = __double2float_rd((double)lo - ldexp(2.0, ex));
}

// One level of the collapse: eight lanes per wide node (fcount[0] nodes in `frontier`; the next level's are
// appended to `next` and counted in fcount[1], once it is known that there is room for them: what is counted
// has been written, and is at most node_cap entries).  A level of a build that has gone wrong (the error
// word) does nothing; one that runs out of nodes shows in counters[0] (scene_build).  What bounds it: the chain of dependent loads of the cost
// decisions and the copies of leaf triangles; the first levels are too small to fill the GPU, so a
// node's own latency counts.  With one thread per node (736 bytes of local arrays) a level took 133 us
// on 500 k triangles, 1061 us in all; with eight lanes 205 us in all.
constexpr int COLLAPSE_BLOCK = 128;
constexpr uint32_t COLLAPSE_MAX_LEVELS = 200;
constexpr int ALL_TRIS = 0x7FFFFFFF;   // frontier entry of a scene of at most 3 triangles: one leaf

__global__ void __launch_bounds__(COLLAPSE_BLOCK) k_collapse(CollapseArgs A, const int2* __restrict__ frontier,
                                                             uint32_t* __restrict__ fcount, int2* __restrict__ next) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    __shared__ int2 s_open[COLLAPSE_BLOCK];        // subtree and slots handed to another lane
    __shared__ int s_child[COLLAPSE_BLOCK];        // lane of the child that a slot takes
    const int lane = threadIdx.x & 31, oct0 = lane & 24, sub = lane & 7;
    const int tid0 = threadIdx.x & ~7;
    const uint32_t octs = gridDim.x * (COLLAPSE_BLOCK / 8), todo = *fcount;
    const int n = A.n;
    auto oct_ballot = [&](bool b) { return (__ballot_sync(ALL, b) >> oct0) & 0xFFu; };
    auto from = [&](auto v, int k) { return __shfl_sync(ALL, v, oct0 + k); };
    if (__any_sync(ALL, *A.err != 0u)) return;
    // the warp's four nodes go through every step together (the trip count is uniform over the warp)
    const uint32_t t0 = (blockIdx.x * COLLAPSE_BLOCK + threadIdx.x) / 32u * 4u;
    for (uint32_t tw = t0; tw < todo; tw += octs) {
        const uint32_t t = tw + (uint32_t)(lane >> 3);
        const bool live = t < todo;
        const int2 job = live ? frontier[t] : make_int2(0, 0);
        const uint32_t wnode = (uint32_t)job.y;

        // expand by the cost decisions: lane `sub` holds subtree `ref` with k slots (k 0: none), which
        // occupies slots sub .. sub + k - 1; a subtree stays one child (a leaf or an 8-wide node) unless
        // spreading its k slots over its own children is cheaper
        int ref = job.x, k = live && sub == 0 && n > 0 ? 8 : 0;
        bool open = k > 0 && ref != ALL_TRIS;   // the node itself is always opened
        while (__any_sync(ALL, open)) {
            s_open[threadIdx.x] = make_int2(0, 0);
            __syncwarp();
            if (open) {
                const int2 c = A.child[ref];
                float cl[9], cr[9];
                dp_child(A.dp, c.x, c.x < 0 ? box_area(A.nbox[2 * box_index(n, c.x)], A.nbox[2 * box_index(n, c.x) + 1]) : 0.f,
                         A.cost_tri, cl);
                dp_child(A.dp, c.y, c.y < 0 ? box_area(A.nbox[2 * box_index(n, c.y)], A.nbox[2 * box_index(n, c.y) + 1]) : 0.f,
                         A.cost_tri, cr);
                int bk = 1;
                float best = 3.0e38f;
#pragma unroll
                for (int kt = 2; kt <= 8; ++kt) {   // k as a constant, so that cl and cr stay in registers
                    if (kt != k) continue;
#pragma unroll
                    for (int kk = 1; kk < kt; ++kk) {
                        const float v = cl[kk] + cr[kt - kk];
                        if (v < best) {
                            best = v;
                            bk = kk;
                        }
                    }
                }
                s_open[tid0 + sub + bk] = make_int2(c.y, k - bk);
                ref = c.x;
                k = bk;
            }
            __syncwarp();
            const int2 given = s_open[threadIdx.x];
            if (given.y) {
                ref = given.x;
                k = given.y;
            }
            open = (open || given.y) && ref >= 0 && k > 1 && __ldg(A.dp + 8ull * ref + k - 1) < __ldg(A.dp + 8ull * ref);
            __syncwarp();
        }

        // the lane's child: box, number of triangles, first sorted position
        const bool child = k > 0;
        const uint32_t cmask = oct_ballot(child);
        const int rank = __popc(cmask & ((1u << sub) - 1u));
        float clo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, chi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
        int cnt = 0, first = 0;
        bool bad = false;
        if (child) {
            size_t bi;
            if (ref == ALL_TRIS) {
                cnt = n;
                bi = n > 1 ? 0 : (size_t)(n - 1);   // root box (internal 0) or the single leaf
            } else {
                const int2 r = ref >= 0 ? A.range[ref] : make_int2(~ref, ~ref);
                cnt = r.y - r.x + 1;
                first = r.x;
                bi = box_index(n, ref);
                bad = cnt < 1 || first < 0 || first + cnt > n;   // damaged ranges: report, read nothing
            }
            if (!bad) {
                const float4 a = A.nbox[2 * bi], b = A.nbox[2 * bi + 1];
                clo[0] = a.x; clo[1] = a.y; clo[2] = a.z;
                chi[0] = b.x; chi[1] = b.y; chi[2] = b.z;
            }
        }
        const bool node_bad = oct_ballot(bad) != 0u;
        if (node_bad && sub == 0) atomicOr(A.err, (uint32_t)DEVERR_BUILD_OVERFLOW);
        float lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = clo[a];
            hi[a] = chi[a];
            for (int o = 1; o < 8; o <<= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(ALL, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(ALL, hi[a], o));
            }
            if (!cmask) lo[a] = hi[a] = 0.f;
        }

        // slot assignment: slot s takes the child whose centroid lies farthest along
        // D(s) = (s&1 ? -1 : 1, s&2 ? -1 : 1, s&4 ? -1 : 1) from the node centre (greedy; of equal scores
        // the first child, then the first slot)
        const float ox = 0.5f * (clo[0] + chi[0]) - 0.5f * (lo[0] + hi[0]);
        const float oy = 0.5f * (clo[1] + chi[1]) - 0.5f * (lo[1] + hi[1]);
        const float oz = 0.5f * (clo[2] + chi[2]) - 0.5f * (lo[2] + hi[2]);
        uint32_t free_slots = 0xFFu;
        int slot = -1;
        s_child[threadIdx.x] = -1;
        __syncwarp();
        for (int it = 0; it < 8; ++it) {
            float best = -3.4e38f;
            int what = 64;   // child's rank x 8 + slot
            if (child && slot < 0) {
                int bs = __ffs(free_slots) - 1;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float v = ((s & 1) ? -ox : ox) + ((s & 2) ? -oy : oy) + ((s & 4) ? -oz : oz);
                    if (((free_slots >> s) & 1u) && v > best) {
                        best = v;
                        bs = s;
                    }
                }
                what = rank * 8 + bs;
            }
            for (int o = 1; o < 8; o <<= 1) {
                const float v = __shfl_xor_sync(ALL, best, o);
                const int w = __shfl_xor_sync(ALL, what, o);
                if (v > best || (v == best && w < what)) {
                    best = v;
                    what = w;
                }
            }
            if (what < 64) {
                free_slots &= ~(1u << (what & 7));
                if (child && slot < 0 && rank == (what >> 3)) slot = what & 7;
            }
        }
        if (slot >= 0) s_child[tid0 + slot] = sub;
        __syncwarp();

        // from here lane `sub` is slot `sub`
        const int src = s_child[threadIdx.x];
        const bool full = src >= 0 && !node_bad;
        const int from_lane = max(src, 0);
        ref = from(ref, from_lane);
        cnt = from(cnt, from_lane);
        if (!full) cnt = 0;
        first = from(first, from_lane);
        for (int a = 0; a < 3; ++a) {
            clo[a] = from(clo[a], from_lane);
            chi[a] = from(chi[a], from_lane);
        }
        const bool leaf = full && cnt <= 3, inner = full && cnt > 3;
        const uint32_t imask = oct_ballot(inner);
        const int irank = __popc(imask & ((1u << sub) - 1u));
        const uint32_t n_int = __popc(imask);
        uint32_t tri_off = leaf ? (uint32_t)cnt : 0u;   // triangles of the leaves in lower slots
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t v = __shfl_up_sync(ALL, tri_off, o, 8);
            if (sub >= o) tri_off += v;
        }
        const uint32_t n_tri = from(tri_off, 7);
        tri_off -= leaf ? (uint32_t)cnt : 0u;
        uint32_t child_base = 0, tri_base = 0, next_base = 0;
        if (sub == 0) {
            if (n_int) child_base = atomicAdd(&A.counters[0], n_int);
            if (n_tri) tri_base = atomicAdd(&A.counters[1], n_tri);
        }
        child_base = from(child_base, 0);
        tri_base = from(tri_base, 0);
        const bool placed = tri_base + n_tri <= (uint32_t)n;
        if (!placed && sub == 0) atomicOr(A.err, (uint32_t)DEVERR_BUILD_OVERFLOW);
        const bool write = live && !node_bad && placed && child_base + n_int <= A.node_cap;
        if (write && sub == 0 && n_int) next_base = atomicAdd(&fcount[1], n_int);
        next_base = from(next_base, 0);

        // child planes in quanta; lane a finds the grid of axis a
        float p[3];
        int ex[3];
        {
            float pa = 0.f;
            int ea = 0;
            if (sub < 3) node_grid(sub == 0 ? lo[0] : sub == 1 ? lo[1] : lo[2], sub == 0 ? hi[0] : sub == 1 ? hi[1] : hi[2], pa, ea);
            for (int a = 0; a < 3; ++a) {
                p[a] = from(pa, a);
                ex[a] = from(ea, a);
            }
        }
        uint32_t q[6];   // lo x, y, z, hi x, y, z
        for (int a = 0; a < 3; ++a) {
            q[a] = 0xFFu;
            q[3 + a] = 0u;
            if (!full) continue;
            const double iq = ldexp(1.0, -ex[a]);   // 1 / 2^ex, exact: the products equal the quotients
            const bool even = !(sub & 1);
            const double l = plane_below(((double)clo[a] - (double)p[a]) * iq, even);
            const double h = plane_above(((double)chi[a] - (double)p[a]) * iq, even);
            if (l < 0 || h > 255) atomicOr(A.err, (uint32_t)DEVERR_QUANT_RANGE);
            q[a] = (uint32_t)fmax(0.0, fmin(255.0, l));
            q[3 + a] = (uint32_t)fmax(0.0, fmin(255.0, h));
        }
        uint32_t valid = leaf ? ((1u << cnt) - 1u) << (3 * sub) : 0u;
        for (int o = 1; o < 8; o <<= 1) valid |= __shfl_xor_sync(ALL, valid, o);
        uint32_t* const words = reinterpret_cast<uint32_t*>(A.nodes + wnode);
        auto put = [&](uint32_t row, uint32_t word, uint32_t v) {   // rows permuted by node (WideNode)
            if (write) words[4u * (row ^ (wnode & 7u)) + word] = v;
        };
        for (int r = 0; r < 6; ++r) {
            const uint32_t odd = __shfl_xor_sync(ALL, q[r], 1);
            if (!(sub & 1)) put(2u + r, (uint32_t)sub >> 1, plane_word(q[r], odd));
        }
        const uint32_t eword = ((uint32_t)(ex[0] + 127) << 23) | ((uint32_t)(ex[1] + 127) << 15) |
                               ((uint32_t)(ex[2] + 127) << 7);
        const uint32_t head = sub == 0 ? __float_as_uint(p[0]) : sub == 1 ? __float_as_uint(p[1]) : sub == 2 ? __float_as_uint(p[2])
                              : sub == 3 ? eword : sub == 4 ? child_base : sub == 5 ? tri_base : sub == 6 ? valid | (imask << 24) : 0u;
        put((uint32_t)sub >> 2, (uint32_t)sub & 3u, head);
        if (write && inner) next[next_base + irank] = make_int2(ref, (int)(child_base + irank));
        if (write && leaf) {
            for (int m = 0; m < cnt; ++m) {
                const uint32_t at = tri_base + tri_off + m;
                const uint32_t prim = A.sorted[first + m];
                A.tris[3ull * at + 0] = A.geo[3ull * prim + 0];
                A.tris[3ull * at + 1] = A.geo[3ull * prim + 1];
                A.tris[3ull * at + 2] = A.geo[3ull * prim + 2];
                A.leaf_prim[at] = prim;
                A.leaf_entity[at] = A.prim_ent[prim];
                if (A.vn) {
                    A.leaf_vn[3ull * at + 0] = A.vn[3ull * prim + 0];
                    A.leaf_vn[3ull * at + 1] = A.vn[3ull * prim + 1];
                    A.leaf_vn[3ull * at + 2] = A.vn[3ull * prim + 2];
                }
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- binned-SAH topology
// Top-down binned SAH (16 bins on each axis over the centroid bounds; surface area x count) down to
// segments of at most SAH_T triangles, which Karras' construction then builds (its prefix function
// restricted to the segment).  Partitions are stable, so every segment keeps the Morton order of the
// global sort.  Node numbering follows the binary radix tree: a segment [f, l] uses internal
// indices f .. l - 1, and the split that puts [first, p) left and [p, last] right gets index p - 1,
// the last position of its left part, which no segment uses; together that is exactly n - 1 nodes,
// so the collapse consumes the tree unchanged (its root is passed explicitly).
//
// Tasks of more than SAH_SUB triangles are split level by level over the whole GPU (k_sah_bin, k_sah_split,
// k_sah_flags, k_scan, k_sah_scatter per level; the number of a level's tasks stays on the device); a task
// of at most SAH_SUB triangles is taken to its segments by one block (k_sah_subtree).  What bounded the
// build before was latency and atomics: twenty levels of thirteen launches and a host round trip each,
// one thread per task reading 2.5 KB of bins, 39 shared-memory atomics per triangle on the few bins that
// Morton neighbours share.  500 k triangles, levels and segments: about 4.6 -> 1.4 ms with the host's waits (kernels alone 3.6 ->
// 1.05 ms).
constexpr int SAH_BINS = 16;
constexpr int SAH_T = 4;
constexpr int SAH_W = 13;                               // count, box lo/hi, centroid lo/hi (fkeys)
constexpr int SAH_TASK_WORDS = 3 * SAH_BINS * SAH_W;
constexpr int SAH_TILE = 1024;                          // positions per block of the flag and scatter kernels
constexpr int SAH_BIN_TILE = 512;                       // positions per block of the binning kernel
constexpr int SAH_SUB = 512;                            // tasks of at most this many triangles: k_sah_subtree
constexpr int SAH_MAX_LEVELS = 256;
constexpr uint32_t WARP = 0xFFFFFFFFu;

struct SahTask {
    int first, count;
    float clo[3], chi[3];    // centroid bounds
    int parent, side;        // parent split node (-1 for the root) and which child this is
};

struct SahSplit {
    int nl;                  // triangles of the left child
    int axis, bin;           // axis < 0: split by position (no usable centroid extent)
    float clo[2][3], chi[2][3];   // centroid bounds of the left and right child
};

// what the level kernels share on the device
struct SahState {
    uint32_t n_sub;                        // tasks of k_sah_subtree
    int root;                              // internal index of the root
    uint32_t n_tasks[SAH_MAX_LEVELS + 1];  // tasks of each level
};

struct SahTree {
    int n;
    int2* child;
    int2* range;
    int* parent;
    int *seg_lo, *seg_hi;                  // per position: its segment
};

__device__ __forceinline__ int sah_bin(float c, float lo, float hi) {
    const float ext = hi - lo;
    if (!(ext > 0.f)) return 0;
    const int b = (int)((c - lo) * ((float)SAH_BINS / ext));
    return max(0, min(SAH_BINS - 1, b));
}

// value of bin word w without triangles
__device__ __forceinline__ uint32_t sah_empty(int w) {
    const int k = w % SAH_W;
    return k == 0 ? 0u : (((k - 1) % 6) < 3 ? 0xFFFFFFFFu : 0u);
}

__global__ void k_sah_root(const uint32_t* __restrict__ keys, int n, SahTask* __restrict__ tasks,
                           SahTask* __restrict__ sub, uint32_t* __restrict__ bins, SahState* __restrict__ state) {
    for (int w = threadIdx.x; w < SAH_TASK_WORDS; w += blockDim.x) bins[w] = sah_empty(w);
    for (int l = threadIdx.x; l <= SAH_MAX_LEVELS; l += blockDim.x) state->n_tasks[l] = l == 0 && n > SAH_SUB ? 1u : 0u;
    if (threadIdx.x) return;
    SahTask r;
    r.first = 0;
    r.count = n;
    for (int k = 0; k < 3; ++k) {
        r.clo[k] = fkey_inv(keys[6 + k]);
        r.chi[k] = fkey_inv(keys[9 + k]);
    }
    r.parent = -1;
    r.side = 0;
    (n > SAH_SUB ? tasks : sub)[0] = r;
    state->n_sub = n > SAH_SUB ? 0u : 1u;
    state->root = -1;
}

__device__ __forceinline__ void sah_add(uint32_t* b, uint32_t cnt, const uint32_t key[12]) {
    atomicAdd(&b[0], cnt);
    for (int k = 0; k < 3; ++k) {
        atomicMin(&b[1 + k], key[k]);
        atomicMax(&b[4 + k], key[3 + k]);
        atomicMin(&b[7 + k], key[6 + k]);
        atomicMax(&b[10 + k], key[9 + k]);
    }
}

// Adds the warp's triangles (lanes in `on`) to the bins of their task in shared memory.  Morton neighbours
// share bins: where the warp's lanes fall into few combinations of bins, the lanes of each are first
// reduced to one (counts, minima and maxima do not depend on the order of the additions); past
// SAH_GROUPS combinations, which run one after the other, the lanes' own atomics are faster.
constexpr int SAH_GROUPS = 3;
__device__ __forceinline__ void sah_bin_warp(uint32_t* bins, bool on, const float lo[3], const float hi[3],
                                             const float c[3], const float clo[3], const float chi[3]) {
    const uint32_t active = __ballot_sync(WARP, on);
    if (on) {
        int b[3];
        uint32_t key[12];
        for (int a = 0; a < 3; ++a) {
            b[a] = sah_bin(c[a], clo[a], chi[a]);
            key[a] = fkey(lo[a]);
            key[3 + a] = fkey(hi[a]);
            key[6 + a] = key[9 + a] = fkey(c[a]);
        }
        const uint32_t peers = __match_any_sync(active, b[0] | b[1] << 8 | b[2] << 16);
        const bool leader = (int)(threadIdx.x & 31) == __ffs(peers) - 1;
        uint32_t cnt = 1;
        bool add = true;
        if (__popc(__ballot_sync(active, leader)) <= SAH_GROUPS) {
            for (int k = 0; k < 12; ++k)
                key[k] = k % 6 < 3 ? __reduce_min_sync(peers, key[k]) : __reduce_max_sync(peers, key[k]);
            cnt = (uint32_t)__popc(peers);
            add = leader;
        }
        if (add)
            for (int a = 0; a < 3; ++a) sah_add(bins + (a * SAH_BINS + b[a]) * SAH_W, cnt, key);
    }
    __syncwarp();
}

// One block per SAH_BIN_TILE positions: each task with positions in the tile (a contiguous range) is binned in
// shared memory, then added to the task's bins.
__global__ void __launch_bounds__(SAH_BIN_TILE / 2) k_sah_bin(const uint32_t* __restrict__ perm, const int* __restrict__ task_of,
                                                 const SahTask* __restrict__ tasks,
                                                 const uint32_t* __restrict__ n_tasks, const float4* __restrict__ tbox,
                                                 const float4* __restrict__ cen, int n, uint32_t* __restrict__ bins) {
    __shared__ uint32_t sb[SAH_TASK_WORDS];
    __shared__ int s_next;
    if (!*n_tasks) return;
    const int b0 = blockIdx.x * SAH_BIN_TILE, b1 = min(n, b0 + SAH_BIN_TILE);
    for (int p = b0; p < b1;) {
        const int t = task_of[p];   // the same for every thread
        if (t < 0) {                // finished positions: to the next one with a task
            __syncthreads();
            if (threadIdx.x == 0) s_next = b1;
            __syncthreads();
            int q = b1;
            for (int i = p + threadIdx.x; i < b1; i += blockDim.x)
                if (task_of[i] >= 0) {
                    q = i;
                    break;
                }
            if (q < b1) atomicMin(&s_next, q);
            __syncthreads();
            p = s_next;
            continue;
        }
        const SahTask T = tasks[t];
        const int e = min(b1, T.first + T.count);
        for (int w = threadIdx.x; w < SAH_TASK_WORDS; w += blockDim.x) sb[w] = sah_empty(w);
        __syncthreads();
        for (int i0 = p; i0 < e; i0 += blockDim.x) {
            const int i = i0 + threadIdx.x;
            const bool on = i < e;
            float lo[3], hi[3], c[3];
            if (on) {
                const uint32_t q = perm[i];
                const float4 l = tbox[2ull * q], h = tbox[2ull * q + 1], m = cen[q];
                lo[0] = l.x; lo[1] = l.y; lo[2] = l.z;
                hi[0] = h.x; hi[1] = h.y; hi[2] = h.z;
                c[0] = m.x; c[1] = m.y; c[2] = m.z;
            }
            sah_bin_warp(sb, on, lo, hi, c, T.clo, T.chi);
        }
        __syncthreads();
        uint32_t* g = bins + (size_t)t * SAH_TASK_WORDS;
        for (int w = threadIdx.x; w < SAH_TASK_WORDS; w += blockDim.x) {
            const int k = w % SAH_W;
            const uint32_t v = sb[w];
            if (v == sah_empty(w)) continue;
            if (k == 0) atomicAdd(&g[w], v);
            else if (((k - 1) % 6) < 3) atomicMin(&g[w], v);
            else atomicMax(&g[w], v);
        }
        __syncthreads();
        p = e;
    }
}

__device__ __forceinline__ float sah_area(const float lo[3], const float hi[3]) {
    const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// The cheapest of the 3 x 15 bin boundaries by surface area x count (of equal ones the first axis, then the
// first boundary), by one warp: a lane per bin, two axes at a time; prefix and suffix boxes by shuffles.
__device__ __forceinline__ SahSplit sah_best_split(const uint32_t* B, const SahTask& T) {
    const int lane = threadIdx.x & 31, bin = lane & 15;
    float best = 3.0e38f;
    int where = 1 << 20;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const int a = 2 * pass + (lane >> 4);
        uint32_t cnt = 0;
        float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
        if (a < 3) {
            const uint32_t* w = B + (a * SAH_BINS + bin) * SAH_W;
            cnt = w[0];
            if (cnt)
                for (int k = 0; k < 3; ++k) {
                    lo[k] = fkey_inv(w[1 + k]);
                    hi[k] = fkey_inv(w[4 + k]);
                }
        }
        uint32_t lc = cnt, rc = cnt;   // bins [0, bin], bins [bin, 16)
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int k = 0; k < 3; ++k) {
            llo[k] = rlo[k] = lo[k];
            lhi[k] = rhi[k] = hi[k];
        }
        for (int o = 1; o < 16; o <<= 1) {
            const uint32_t uc = __shfl_up_sync(WARP, lc, o, 16), dc = __shfl_down_sync(WARP, rc, o, 16);
            if (bin >= o) lc += uc;
            if (bin + o < 16) rc += dc;
            for (int k = 0; k < 3; ++k) {   // a lane without a source gets its own value back
                llo[k] = fminf(llo[k], __shfl_up_sync(WARP, llo[k], o, 16));
                lhi[k] = fmaxf(lhi[k], __shfl_up_sync(WARP, lhi[k], o, 16));
                rlo[k] = fminf(rlo[k], __shfl_down_sync(WARP, rlo[k], o, 16));
                rhi[k] = fmaxf(rhi[k], __shfl_down_sync(WARP, rhi[k], o, 16));
            }
        }
        // boundary `bin`: bins below it left, the others right
        lc = __shfl_up_sync(WARP, lc, 1, 16);
        for (int k = 0; k < 3; ++k) {
            llo[k] = __shfl_up_sync(WARP, llo[k], 1, 16);
            lhi[k] = __shfl_up_sync(WARP, lhi[k], 1, 16);
        }
        const float ext = a == 0 ? T.chi[0] - T.clo[0] : a == 1 ? T.chi[1] - T.clo[1] : T.chi[2] - T.clo[2];
        if (a < 3 && bin >= 1 && ext > 0.f && lc && rc) {
            const float c = __fmaf_rn(sah_area(llo, lhi), (float)lc, __fmul_rn(sah_area(rlo, rhi), (float)rc));
            if (c < best) {
                best = c;
                where = a * SAH_BINS + bin;
            }
        }
    }
    for (int o = 1; o < 32; o <<= 1) {
        const float c = __shfl_xor_sync(WARP, best, o);
        const int v = __shfl_xor_sync(WARP, where, o);
        if (c < best || (c == best && v < where)) {
            best = c;
            where = v;
        }
    }
    SahSplit S;
    if (where == 1 << 20) {
        S.nl = T.count / 2;
        S.axis = -1;
        S.bin = 0;
        for (int k = 0; k < 3; ++k) {
            S.clo[0][k] = S.clo[1][k] = T.clo[k];
            S.chi[0][k] = S.chi[1][k] = T.chi[k];
        }
        return S;
    }
    S.axis = where / SAH_BINS;
    S.bin = where % SAH_BINS;
    const uint32_t* w = B + (S.axis * SAH_BINS + bin) * SAH_W;
    const bool left = bin < S.bin;
    S.nl = (int)__reduce_add_sync(WARP, lane < 16 && left ? w[0] : 0u);
    for (int k = 0; k < 3; ++k) {   // empty bins hold the neutral keys
        S.clo[0][k] = fkey_inv(__reduce_min_sync(WARP, left ? w[7 + k] : 0xFFFFFFFFu));
        S.clo[1][k] = fkey_inv(__reduce_min_sync(WARP, left ? 0xFFFFFFFFu : w[7 + k]));
        S.chi[0][k] = fkey_inv(__reduce_max_sync(WARP, left ? w[10 + k] : 0u));
        S.chi[1][k] = fkey_inv(__reduce_max_sync(WARP, left ? 0u : w[10 + k]));
    }
    return S;
}

// Split node of a task, by one lane: its range and links
__device__ __forceinline__ int sah_node(const SahTree& tree, int first, int count, int nl, int parent, int side) {
    const int X = first + nl - 1;
    tree.range[X] = make_int2(first, first + count - 1);
    tree.parent[X] = parent;
    if (parent >= 0) {
        if (side == 0) tree.child[parent].x = X;
        else tree.child[parent].y = X;
    }
    return X;
}

// Final segment [first, first + count) under split node `parent`, by one lane
__device__ __forceinline__ void sah_segment(const SahTree& tree, int first, int count, int parent, int side) {
    for (int p = first; p < first + count; ++p) {
        tree.seg_lo[p] = first;
        tree.seg_hi[p] = first + count - 1;
    }
    const int root = count >= 2 ? first : ~first;
    if (side == 0) tree.child[parent].x = root;
    else tree.child[parent].y = root;
    tree.parent[root >= 0 ? root : (tree.n - 1) + ~root] = parent;
}

// where a task of a level sends its triangles
struct SahMove {
    int nl, axis, bin;
    int next[2];             // task of the next level of each child, -1: none
    uint32_t before;         // left triangles before the task's first position in its tile (k_sah_flags)
};

// One warp per task of a level: its split, the node, and its children: tasks of the next level (bins
// cleared), tasks of k_sah_subtree, or segments.
__global__ void __launch_bounds__(128) k_sah_split(SahTree tree, const SahTask* __restrict__ tasks, int level,
                                                   SahState* __restrict__ state, const uint32_t* __restrict__ bins,
                                                   SahMove* __restrict__ moves, SahTask* __restrict__ next,
                                                   uint32_t* __restrict__ next_bins, SahTask* __restrict__ sub) {
    const int lane = threadIdx.x & 31;
    const uint32_t todo = state->n_tasks[level], warps = gridDim.x * 4;
    for (uint32_t t = blockIdx.x * 4 + (threadIdx.x >> 5); t < todo; t += warps) {
        const SahTask T = tasks[t];
        const SahSplit S = sah_best_split(bins + (size_t)t * SAH_TASK_WORDS, T);
        int X = 0, slot[2] = {-1, -1};
        if (lane == 0) {
            X = sah_node(tree, T.first, T.count, S.nl, T.parent, T.side);
            if (T.parent < 0) state->root = X;
        }
        for (int side = 0; side < 2; ++side) {
            SahTask C;
            C.first = side ? T.first + S.nl : T.first;
            C.count = side ? T.count - S.nl : S.nl;
            for (int k = 0; k < 3; ++k) {
                C.clo[k] = S.clo[side][k];
                C.chi[k] = S.chi[side][k];
            }
            C.parent = X;
            C.side = side;
            if (C.count > SAH_SUB) {
                if (lane == 0) {
                    slot[side] = (int)atomicAdd(&state->n_tasks[level + 1], 1u);
                    next[slot[side]] = C;
                }
                slot[side] = __shfl_sync(WARP, slot[side], 0);
                for (int w = lane; w < SAH_TASK_WORDS; w += 32) next_bins[(size_t)slot[side] * SAH_TASK_WORDS + w] = sah_empty(w);
            } else if (lane == 0) {
                if (C.count > SAH_T) sub[atomicAdd(&state->n_sub, 1u)] = C;
                else sah_segment(tree, C.first, C.count, X, side);
            }
        }
        if (lane == 0) moves[t] = SahMove{S.nl, S.axis, S.bin, {slot[0], slot[1]}, 0u};
    }
}

__device__ __forceinline__ bool sah_left(const SahTask& T, const SahMove& S, int i, const float4& c) {
    if (S.axis < 0) return i - T.first < S.nl;
    const float v = S.axis == 0 ? c.x : S.axis == 1 ? c.y : c.z;
    return sah_bin(v, T.clo[S.axis], T.chi[S.axis]) < S.bin;
}

// Exclusive prefix over the words of left flags of a block (at most 32, in shared memory), by one warp;
// returns their number of left flags.
constexpr int SAH_WORDS = SAH_TILE / 32;
static_assert(SAH_WORDS == 32 && SAH_SUB <= SAH_TILE, "one word per lane");
__device__ __forceinline__ uint32_t sah_word_scan(const uint32_t* words, int n_words, uint32_t* prefix) {
    const int lane = threadIdx.x & 31;
    const uint32_t v = lane < n_words ? (uint32_t)__popc(words[lane]) : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(WARP, x, o);
        if (lane >= o) x += y;
    }
    prefix[lane] = x - v;
    return __shfl_sync(WARP, x, 31);
}

__global__ void __launch_bounds__(256) k_sah_flags(const uint32_t* __restrict__ perm, const int* __restrict__ task_of,
                                                   const SahTask* __restrict__ tasks,
                                                   const uint32_t* __restrict__ n_tasks, SahMove* __restrict__ moves,
                                                   const float4* __restrict__ cen, int n, uint32_t* __restrict__ flags,
                                                   uint32_t* __restrict__ tile_total) {
    __shared__ uint32_t words[SAH_WORDS], prefix[SAH_WORDS];
    if (!*n_tasks) return;
    const int b0 = blockIdx.x * SAH_TILE, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t firsts = 0;   // of this thread's positions, those that begin a task
#pragma unroll
    for (int j = 0; j < SAH_TILE / 256; ++j) {
        const int i = b0 + j * 256 + threadIdx.x;
        bool left = false;
        if (i < n) {
            const int t = task_of[i];
            if (t >= 0) {
                const SahTask& T = tasks[t];
                left = sah_left(T, moves[t], i, cen[perm[i]]);
                if (i == T.first) firsts |= 1u << j;
            }
        }
        const uint32_t m = __ballot_sync(WARP, left);
        if (lane == 0) words[j * 8 + warp] = flags[(size_t)blockIdx.x * SAH_WORDS + j * 8 + warp] = m;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t total = sah_word_scan(words, SAH_WORDS, prefix);
        if (lane == 0) tile_total[blockIdx.x] = total;
    }
    __syncthreads();
    for (int j = 0; j < SAH_TILE / 256; ++j)
        if ((firsts >> j) & 1u)
            moves[task_of[b0 + j * 256 + threadIdx.x]].before = prefix[j * 8 + warp] +
                                                               (uint32_t)__popc(words[j * 8 + warp] & ((1u << lane) - 1u));
}

// Stable partition of every task's range; finished positions move along.
__global__ void __launch_bounds__(256) k_sah_scatter(const uint32_t* __restrict__ perm_in, uint32_t* __restrict__ perm_out,
                                                     const int* __restrict__ task_in, int* __restrict__ task_out,
                                                     const SahTask* __restrict__ tasks,
                                                     const uint32_t* __restrict__ n_tasks,
                                                     const SahMove* __restrict__ moves, int n,
                                                     const uint32_t* __restrict__ flags,
                                                     const uint32_t* __restrict__ tile_first) {
    __shared__ uint32_t words[SAH_WORDS], prefix[SAH_WORDS];
    if (!*n_tasks) return;
    const int b0 = blockIdx.x * SAH_TILE, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        words[lane] = flags[(size_t)blockIdx.x * SAH_WORDS + lane];
        __syncwarp();
        sah_word_scan(words, SAH_WORDS, prefix);
    }
    __syncthreads();
    const uint32_t here = tile_first[blockIdx.x];
#pragma unroll
    for (int j = 0; j < SAH_TILE / 256; ++j) {
        const int i = b0 + j * 256 + threadIdx.x;
        if (i >= n) break;
        const int t = task_in[i];
        int pos = i, to = -1;
        if (t >= 0) {
            const SahMove& S = moves[t];
            const int f = tasks[t].first;
            const uint32_t m = words[j * 8 + warp];
            const uint32_t scan = here + prefix[j * 8 + warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
            const int lr = (int)(scan - (tile_first[f / SAH_TILE] + S.before));   // left triangles before i in the task
            const bool left = (m >> lane) & 1u;
            pos = left ? f + lr : f + S.nl + (i - f - lr);
            to = S.next[left ? 0 : 1];
        }
        perm_out[pos] = perm_in[i];
        task_out[pos] = to;
    }
}

// One block takes a task of at most SAH_SUB triangles to its segments: boxes, centroids and the order in
// shared memory.  Per level, tasks of more than SUB_WIDE triangles are taken by all warps, one after the
// other, the rest by a warp each.  The task's part of `sorted` is read first and rewritten segment by
// segment.
struct SubTask {
    float clo[3], chi[3];
    int parent;
    uint16_t first, count;   // within the block's task
    uint16_t side, pad;
};
constexpr int SUB_TASKS = SAH_SUB / (SAH_T + 1) + 1, SUB_WARPS = 8, SUB_WIDE = 96;
struct SubShared {
    float lo[3][SAH_SUB], hi[3][SAH_SUB], c[3][SAH_SUB];
    uint32_t prim[SAH_SUB];
    uint32_t bins[SUB_WARPS][SAH_TASK_WORDS];
    SubTask tasks[2][SUB_TASKS];
    SahSplit split;
    uint32_t words[32], prefix[32];
    uint16_t order[2][SAH_SUB];
    uint32_t n_tasks[2];
};

// The split node of a block-local task and its children, by one warp, after the task's part of order[cur ^ 1]
// has been written
__device__ __forceinline__ void sub_children(SubShared& M, const SahTree& tree, SahState* state, uint32_t* sorted,
                                             int block_first, int cur, const SahTask& T, const SahSplit& S) {
    const int lane = threadIdx.x & 31;
    int X = 0;
    if (lane == 0) {
        X = sah_node(tree, block_first + T.first, T.count, S.nl, T.parent, T.side);
        if (T.parent < 0) state->root = X;
    }
    for (int sd = 0; sd < 2; ++sd) {
        const int f = sd ? T.first + S.nl : T.first, cnt = sd ? T.count - S.nl : S.nl;
        if (cnt > SAH_T) {
            if (lane == 0) {
                SubTask& C = M.tasks[cur ^ 1][atomicAdd(&M.n_tasks[cur ^ 1], 1u)];
                for (int k = 0; k < 3; ++k) {
                    C.clo[k] = S.clo[sd][k];
                    C.chi[k] = S.chi[sd][k];
                }
                C.parent = X;
                C.first = (uint16_t)f;
                C.count = (uint16_t)cnt;
                C.side = (uint16_t)sd;
            }
        } else {
            if (lane < cnt) sorted[block_first + f + lane] = M.prim[M.order[cur ^ 1][f + lane]];
            if (lane == 0) sah_segment(tree, block_first + f, cnt, X, sd);
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(32 * SUB_WARPS) k_sah_subtree(SahTree tree, const SahTask* __restrict__ sub,
                                                                SahState* __restrict__ state,
                                                                const float4* __restrict__ tbox,
                                                                const float4* __restrict__ cen, uint32_t* sorted) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    SubShared& M = *reinterpret_cast<SubShared*>(sub_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    auto task = [&](int cur, uint32_t t) {
        const SubTask& U = M.tasks[cur][t];
        SahTask T;
        for (int k = 0; k < 3; ++k) {
            T.clo[k] = U.clo[k];
            T.chi[k] = U.chi[k];
        }
        T.first = U.first;
        T.count = U.count;
        T.parent = U.parent;
        T.side = U.side;
        return T;
    };
    // bins the 32 positions from i0 of task T (order[cur]) with one warp
    auto bin_chunk = [&](uint32_t* bins, int cur, const SahTask& T, int i0) {
        const bool on = i0 + lane < T.count;
        float lo[3], hi[3], c[3];
        if (on) {
            const int q = M.order[cur][T.first + i0 + lane];
            for (int k = 0; k < 3; ++k) {
                lo[k] = M.lo[k][q];
                hi[k] = M.hi[k][q];
                c[k] = M.c[k][q];
            }
        }
        sah_bin_warp(bins, on, lo, hi, c, T.clo, T.chi);
    };
    // item and left flag of position i0 + lane
    auto side_of = [&](int cur, const SahTask& T, const SahSplit& S, int i0, int& q) {
        q = 0;
        if (i0 + lane >= T.count) return false;
        q = M.order[cur][T.first + i0 + lane];
        if (S.axis < 0) return i0 + lane < S.nl;
        const float lo = S.axis == 0 ? T.clo[0] : S.axis == 1 ? T.clo[1] : T.clo[2];
        const float hi = S.axis == 0 ? T.chi[0] : S.axis == 1 ? T.chi[1] : T.chi[2];
        return sah_bin(M.c[S.axis][q], lo, hi) < S.bin;
    };
    const uint32_t todo = state->n_sub;
    for (uint32_t item = blockIdx.x; item < todo; item += gridDim.x) {
        const SahTask R = sub[item];
        for (int i = threadIdx.x; i < R.count; i += blockDim.x) {
            const uint32_t p = sorted[R.first + i];
            const float4 l = tbox[2ull * p], h = tbox[2ull * p + 1], m = cen[p];
            M.prim[i] = p;
            M.lo[0][i] = l.x; M.lo[1][i] = l.y; M.lo[2][i] = l.z;
            M.hi[0][i] = h.x; M.hi[1][i] = h.y; M.hi[2][i] = h.z;
            M.c[0][i] = m.x; M.c[1][i] = m.y; M.c[2][i] = m.z;
            M.order[0][i] = (uint16_t)i;
        }
        if (threadIdx.x == 0) {
            SubTask& T = M.tasks[0][0];
            for (int k = 0; k < 3; ++k) {
                T.clo[k] = R.clo[k];
                T.chi[k] = R.chi[k];
            }
            T.parent = R.parent;
            T.first = 0;
            T.count = (uint16_t)R.count;
            T.side = (uint16_t)R.side;
            M.n_tasks[0] = 1;
            M.n_tasks[1] = 0;
        }
        __syncthreads();
        for (int cur = 0; M.n_tasks[cur]; cur ^= 1) {
            const uint32_t nt = M.n_tasks[cur];
            for (uint32_t t = 0; t < nt; ++t) {   // wide tasks: the whole block
                if (M.tasks[cur][t].count <= SUB_WIDE) continue;
                const SahTask T = task(cur, t);
                for (int w = threadIdx.x; w < SAH_TASK_WORDS; w += blockDim.x) M.bins[0][w] = sah_empty(w);
                __syncthreads();
                for (int i0 = 32 * warp; i0 < T.count; i0 += 32 * SUB_WARPS) bin_chunk(M.bins[0], cur, T, i0);
                __syncthreads();
                if (warp == 0) {
                    const SahSplit S = sah_best_split(M.bins[0], T);
                    if (lane == 0) M.split = S;
                }
                __syncthreads();
                const SahSplit S = M.split;
                for (int i0 = 32 * warp; i0 < T.count; i0 += 32 * SUB_WARPS) {
                    int q;
                    const uint32_t m = __ballot_sync(WARP, side_of(cur, T, S, i0, q));
                    if (lane == 0) M.words[i0 / 32] = m;
                }
                __syncthreads();
                if (warp == 0) sah_word_scan(M.words, (T.count + 31) / 32, M.prefix);
                __syncthreads();
                for (int i0 = 32 * warp; i0 < T.count; i0 += 32 * SUB_WARPS) {
                    const int i = i0 + lane;
                    if (i >= T.count) continue;
                    const uint32_t m = M.words[i0 / 32];
                    const int lr = (int)(M.prefix[i0 / 32] + (uint32_t)__popc(m & lt));
                    M.order[cur ^ 1][T.first + ((m >> lane) & 1u ? lr : S.nl + (i - lr))] = M.order[cur][T.first + i];
                }
                __syncthreads();
                if (warp == 0) sub_children(M, tree, state, sorted, R.first, cur, T, S);
            }
            __syncthreads();
            for (uint32_t t = warp; t < nt; t += SUB_WARPS) {
                if (M.tasks[cur][t].count > SUB_WIDE) continue;
                const SahTask T = task(cur, t);
                uint32_t* bins = M.bins[warp];
                for (int w = lane; w < SAH_TASK_WORDS; w += 32) bins[w] = sah_empty(w);
                __syncwarp();
                for (int i0 = 0; i0 < T.count; i0 += 32) bin_chunk(bins, cur, T, i0);
                const SahSplit S = sah_best_split(bins, T);
                int nleft = 0;   // stable partition into the other order
                for (int i0 = 0; i0 < T.count; i0 += 32) {
                    int q;
                    const uint32_t m = __ballot_sync(WARP, side_of(cur, T, S, i0, q));
                    const int lr = nleft + __popc(m & lt);
                    if (i0 + lane < T.count)
                        M.order[cur ^ 1][T.first + ((m >> lane) & 1u ? lr : S.nl + (i0 + lane - lr))] = (uint16_t)q;
                    nleft += __popc(m);
                }
                __syncwarp();
                sub_children(M, tree, state, sorted, R.first, cur, T, S);
            }
            __syncthreads();
            if (threadIdx.x == 0) M.n_tasks[cur] = 0;
            __syncthreads();
        }
        __syncthreads();   // every thread has left the loop before the next task is set up
    }
}

__global__ void k_gather_codes(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ code_by_prim, int n,
                               uint32_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = code_by_prim[perm[i]];
}

__device__ __forceinline__ int delta_seg(const uint32_t* __restrict__ code, int lo, int hi, int i, int j) {
    if (j < lo || j > hi) return -1;
    const uint32_t a = code[i], b = code[j];
    if (a == b) return 32 + __clz((uint32_t)(i ^ j));
    return __clz(a ^ b);
}

// Karras' construction inside each segment [seg_lo, seg_hi] (the last position of a segment is not
// an internal node of it)
__global__ void k_karras_seg(const uint32_t* __restrict__ code, int n, const int* __restrict__ seg_lo,
                             const int* __restrict__ seg_hi, int2* __restrict__ child, int2* __restrict__ range,
                             int* __restrict__ parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int lo_s = seg_lo[i], hi_s = seg_hi[i];
    if (i >= hi_s) return;
    const int d = (delta_seg(code, lo_s, hi_s, i, i + 1) - delta_seg(code, lo_s, hi_s, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta_seg(code, lo_s, hi_s, i, i - d);
    int lmax = 2;
    while (delta_seg(code, lo_s, hi_s, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta_seg(code, lo_s, hi_s, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta_seg(code, lo_s, hi_s, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta_seg(code, lo_s, hi_s, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = (lo == gamma) ? ~gamma : gamma;
    const int right = (hi == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    child[i] = make_int2(left, right);
    range[i] = make_int2(lo, hi);
    parent[left >= 0 ? left : (n - 1) + ~left] = i;
    parent[right >= 0 ? right : (n - 1) + ~right] = i;
}

// Temporaries of sah_topology: about 43 bytes per triangle, which lie where the node boxes and collapse costs
// (96 bytes) come after it (scene_build), so that a context holds no memory for them.
struct SahTemp {
    uint32_t *perm, *flags, *tile, *bins[2], *code;
    int *task_of[2], *seg_lo, *seg_hi;
    SahState* state;
    SahTask *tasks[2], *sub;
    SahMove* moves;
    static uint32_t tiles(size_t n) { return (uint32_t)((n + SAH_TILE - 1) / SAH_TILE); }
    static size_t max_tasks(size_t n) { return n / SAH_SUB + 2; }   // of one level: disjoint ranges of more than SAH_SUB
    // lays them out from mem (null: only the size) and returns the bytes taken
    size_t carve(char* mem, size_t n) {
        size_t off = 0;
        auto take = [&](auto*& q, size_t count) {
            q = mem ? reinterpret_cast<std::remove_reference_t<decltype(q)>>(mem + off) : nullptr;
            off += (count * sizeof(*q) + 255) & ~size_t(255);
        };
        take(perm, n);
        take(task_of[0], n);
        take(task_of[1], n);
        take(flags, (size_t)SAH_WORDS * tiles(n));
        take(tile, tiles(n));
        take(state, 1);
        take(tasks[0], max_tasks(n));
        take(tasks[1], max_tasks(n));
        take(moves, max_tasks(n));
        take(bins[0], SAH_TASK_WORDS * max_tasks(n));
        take(bins[1], SAH_TASK_WORDS * max_tasks(n));
        take(sub, n / (SAH_T + 1) + 2);
        take(seg_lo, n);
        take(seg_hi, n);
        take(code, n);
        return off;
    }
};

// Binned-SAH binary tree over the Morton-sorted triangles (n > SAH_T): fills child / range / parent
// like k_karras, writes the triangle order of the tree's leaves to `sorted` (in place of the Morton order)
// and the root's internal index to *root (device memory).
void sah_topology(crt_context* ctx, int n, const SahTemp& M, const float4* tbox, const float4* cen, const uint32_t* keys,
                  uint32_t* sorted, const uint32_t* code_by_prim, int2* child, int2* range, int* parent, int2* root) {
    cudaStream_t st = ctx->stream;
    const size_t max_tasks = SahTemp::max_tasks(n);
    const uint32_t tiles = SahTemp::tiles(n);
    const uint32_t bin_tiles = (uint32_t)(((size_t)n + SAH_BIN_TILE - 1) / SAH_BIN_TILE);
    uint32_t* const perm[2] = {sorted, M.perm};
    uint32_t *const flags = M.flags, *const tile = M.tile, *const code = M.code;
    int* const* const task_of = M.task_of;
    SahState* const state = M.state;
    SahTask *const *const tasks = M.tasks, *const sub = M.sub;
    SahMove* const moves = M.moves;
    uint32_t* const* const bins = M.bins;
    const SahTree tree{n, child, range, parent, M.seg_lo, M.seg_hi};

    CRT_CUDA(cudaMemsetAsync(task_of[0], 0, 4ull * n, st));   // every position in task 0 (the root)
    k_sah_root<<<1, 256, 0, st>>>(keys, n, tasks[0], sub, bins[0], state);
    check_launch(ctx, "k_sah_root");
    // levels of tasks larger than SAH_SUB: as many as a balanced tree has and three more, then a look
    // at the task counts, then four at a time
    int levels = 0;
    if (n > SAH_SUB) {
        uint32_t h[SAH_MAX_LEVELS + 1];
        int batch = 3;
        for (int m = n; m > SAH_SUB; m = (m + 1) / 2) ++batch;
        for (int launched = 0;;) {
            CRT_CHECK(launched + batch <= SAH_MAX_LEVELS, CRT_ERR_DEVICE, "SAH build did not converge");
            for (int b = 0; b < batch; ++b, ++launched) {
                const int cur = launched & 1, nxt = cur ^ 1;
                const uint32_t* nt = &state->n_tasks[launched];
                k_sah_bin<<<bin_tiles, SAH_BIN_TILE / 2, 0, st>>>(perm[cur], task_of[cur], tasks[cur], nt, tbox, cen, n, bins[cur]);
                check_launch(ctx, "k_sah_bin");
                const size_t bound = std::min<size_t>(launched < 30 ? size_t(1) << launched : max_tasks, max_tasks);
                k_sah_split<<<(uint32_t)std::min<size_t>((bound + 3) / 4, (size_t)ctx->sm_count * 8), 128, 0, st>>>(
                    tree, tasks[cur], launched, state, bins[cur], moves, tasks[nxt], bins[nxt], sub);
                check_launch(ctx, "k_sah_split");
                k_sah_flags<<<tiles, 256, 0, st>>>(perm[cur], task_of[cur], tasks[cur], nt, moves, cen, n, flags, tile);
                check_launch(ctx, "k_sah_flags");
                k_scan<<<1, 1024, 0, st>>>(tile, tiles);
                check_launch(ctx, "k_scan");
                k_sah_scatter<<<tiles, 256, 0, st>>>(perm[cur], perm[nxt], task_of[cur], task_of[nxt], tasks[cur], nt,
                                                     moves, n, flags, tile);
                check_launch(ctx, "k_sah_scatter");
            }
            CRT_CUDA(cudaMemcpyAsync(h, state->n_tasks, sizeof(uint32_t) * (launched + 1), cudaMemcpyDeviceToHost, st));
            CRT_CUDA(cudaStreamSynchronize(st));
            while (levels < launched && h[levels]) ++levels;
            if (!h[launched]) break;
            batch = 4;
        }
    }
    if (levels & 1) CRT_CUDA(cudaMemcpyAsync(sorted, perm[1], 4ull * n, cudaMemcpyDeviceToDevice, st));
    CRT_CUDA(cudaFuncSetAttribute(k_sah_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SubShared)));
    const uint32_t blocks = (uint32_t)std::min<size_t>((size_t)n / 64 + 1, (size_t)ctx->sm_count * 8);
    k_sah_subtree<<<blocks, 32 * SUB_WARPS, sizeof(SubShared), st>>>(tree, sub, state, tbox, cen, sorted);
    check_launch(ctx, "k_sah_subtree");
    CRT_CUDA(cudaMemcpyAsync(&root->x, &state->root, sizeof(int), cudaMemcpyDeviceToDevice, st));
    k_gather_codes<<<(n + 255) / 256, 256, 0, st>>>(sorted, code_by_prim, n, code);
    check_launch(ctx, "k_gather_codes");
    k_karras_seg<<<(n + 254) / 256, 256, 0, st>>>(code, n, tree.seg_lo, tree.seg_hi, child, range, parent);
    check_launch(ctx, "k_karras_seg");
}

inline uint32_t cdiv(size_t a, uint32_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace

// Builds every device array of the scene.  Throws CrtError on failure.
void scene_build(crt_scene* s, const crt_entity_desc* ents, uint32_t n_ents) {
    crt_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    size_t n64 = 0;
    for (uint32_t e = 0; e < n_ents; ++e) n64 += ents[e].n_tris;
    CRT_CHECK(n64 < 0x7FFFFFF0ull, CRT_ERR_INVALID, "scene too large (>= 2^31 triangles)");
    const uint32_t n = (uint32_t)n64;
    s->n_tris = n;
    s->n_entities = n_ents;
    bool any_vn = false;
    for (uint32_t e = 0; e < n_ents; ++e) {
        CRT_CHECK(ents[e].n_tris == 0 || ents[e].tri_xyz, CRT_ERR_INVALID, "entity without triangle data");
        if (ents[e].smooth_shading && ents[e].tri_vn) any_vn = true;
    }

    cudaEvent_t ev0, ev1;
    CRT_CUDA(cudaEventCreate(&ev0));
    CRT_CUDA(cudaEventCreate(&ev1));
    CRT_CUDA(cudaEventRecord(ev0, st));

    // entity table + transforms
    s->host_entities.resize(std::max<uint32_t>(n_ents, 1));
    std::vector<EntXform> xf(std::max<uint32_t>(n_ents, 1));
    uint32_t off = 0;
    for (uint32_t e = 0; e < n_ents; ++e) {
        EntityDev& d = s->host_entities[e];
        std::memcpy(d.color, ents[e].color, sizeof(d.color));
        d.smooth = ents[e].smooth_shading ? 1u : 0u;
        d.id = ents[e].id;
        d.rho_s = ents[e].rho_s;
        d.rho_d = ents[e].rho_d;
        d.pad = 0;
        xf[e].scale = ents[e].scale;
        std::memcpy(xf[e].pos, ents[e].position, sizeof(xf[e].pos));
        std::memcpy(xf[e].rot, ents[e].rotation, sizeof(xf[e].rot));
        xf[e].first = off;
        xf[e].has_vn = (ents[e].smooth_shading && ents[e].tri_vn) ? 1u : 0u;
        off += (uint32_t)ents[e].n_tris;
    }
    CRT_CUDA(cudaMalloc(&s->entities, sizeof(EntityDev) * s->host_entities.size()));
    CRT_CUDA(cudaMemcpyAsync(s->entities, s->host_entities.data(), sizeof(EntityDev) * s->host_entities.size(),
                             cudaMemcpyHostToDevice, st));
    EntXform* d_xf = (EntXform*)ctx_scratch(ctx, SCR_BUILD7, sizeof(EntXform) * xf.size());
    CRT_CUDA(cudaMemcpyAsync(d_xf, xf.data(), sizeof(EntXform) * xf.size(), cudaMemcpyHostToDevice, st));

    const size_t nn = std::max<uint32_t>(n, 1);
    // binned-SAH topology for scenes larger than one segment (the context's build setting), else
    // Karras' radix tree over the Morton order
    const bool sah = ctx->build_sah && n > (uint32_t)SAH_T;
    SahTemp sah_temp;
    // scratch layout
    float* d_xyz = (float*)ctx_scratch(ctx, SCR_BUILD0, nn * 9 * sizeof(float));
    float* d_vnin = any_vn ? (float*)ctx_scratch(ctx, SCR_BUILD1, nn * 9 * sizeof(float)) : nullptr;
    for (uint32_t e = 0; e < n_ents; ++e) {
        if (!ents[e].n_tris) continue;
        const size_t b = (size_t)xf[e].first * 9 * sizeof(float), len = ents[e].n_tris * 9 * sizeof(float);
        CRT_CUDA(cudaMemcpyAsync((char*)d_xyz + b, ents[e].tri_xyz, len, cudaMemcpyDefault, st));
        if (d_vnin) {
            if (xf[e].has_vn) CRT_CUDA(cudaMemcpyAsync((char*)d_vnin + b, ents[e].tri_vn, len, cudaMemcpyDefault, st));
        }
    }
    // one scratch region carved into 256-byte aligned arrays (measured first, then assigned)
    float4 *geo = nullptr, *vn = nullptr, *tbox = nullptr, *cen = nullptr, *nbox = nullptr;
    uint32_t *prim_ent = nullptr, *code_a = nullptr, *idx_a = nullptr, *code_b = nullptr, *idx_b = nullptr;
    uint32_t* code_prim = nullptr;
    float* dpc = nullptr;
    uint32_t *hist = nullptr, *flags = nullptr, *keys = nullptr, *counts = nullptr;
    int2 *child = nullptr, *range = nullptr, *root = nullptr, *front = nullptr, *front_b = nullptr;
    int* parent = nullptr;
    int *tl_cnt = nullptr, *tl_pos = nullptr, *tl_par = nullptr;
    uint32_t* tl_sorted = nullptr;
    const size_t nb_sort = (nn + SORT_TILE - 1) / SORT_TILE;
    auto carve = [&](char* base) {
        size_t off = 0;
        auto take = [&](size_t bytes) {
            off = (off + 255) & ~size_t(255);
            char* p = base ? base + off : nullptr;
            off += bytes;
            return p;
        };
        geo = (float4*)take(nn * 48);
        vn = (float4*)take(any_vn ? nn * 48 : 16);
        prim_ent = (uint32_t*)take(nn * 4);
        tbox = (float4*)take(nn * 32);
        cen = (float4*)take(nn * 16);
        code_a = (uint32_t*)take(nn * 4);
        idx_a = (uint32_t*)take(nn * 4);
        code_prim = (uint32_t*)take(nn * 4);
        code_b = (uint32_t*)take(nn * 4);
        idx_b = (uint32_t*)take(nn * 4);
        hist = (uint32_t*)take(nb_sort * 256 * 4);
        child = (int2*)take(nn * 8);
        range = (int2*)take(nn * 8);
        parent = (int*)take(nn * 8);          // 2n - 1 entries: internal nodes then leaves
        flags = (uint32_t*)take(nn * 4);
        nbox = (float4*)take(nn * 64);        // 2n - 1 nodes x (lo, hi)
        char* const over = base ? (char*)nbox : nullptr;   // sah_topology is done before these two are filled
        const size_t first = off - nn * 64;
        dpc = (float*)take(nn * 32);          // collapse costs: 8 per internal node
        if (sah) off = std::max(off, first + sah_temp.carve(over, nn));
        keys = (uint32_t*)take(64 * 4);
        counts = (uint32_t*)take((2 + COLLAPSE_MAX_LEVELS + 1) * 4);   // collapse: nodes, triangles, nodes per level
        root = (int2*)take(8);                // the collapse's first level: binary root, wide node 0
        front = (int2*)take(nn * 8 + 8);
        front_b = (int2*)take(nn * 8 + 8);
        tl_cnt = (int*)take(nn * 4);
        tl_pos = (int*)take(nn * 8);          // 2n - 1 nodes
        tl_par = (int*)take(nn * 4);
        tl_sorted = (uint32_t*)take(nn * 4);
        return off;
    };
    const size_t total = carve(nullptr);
    carve((char*)ctx_scratch(ctx, SCR_BUILD2, total));

    CRT_CUDA(cudaMemsetAsync(parent, 0xFF, nn * 8, st));
    CRT_CUDA(cudaMemsetAsync(flags, 0, nn * 4, st));

    if (n) {
        k_transform<<<cdiv(n, BLOCK), BLOCK, 0, st>>>(d_xyz, d_vnin, d_xf, n_ents, n, geo, any_vn ? vn : nullptr,
                                                      prim_ent, tbox, cen);
        check_launch(ctx, "k_transform");
        uint32_t init[12];
        for (int k = 0; k < 12; ++k) init[k] = (k % 6) < 3 ? 0xFFFFFFFFu : 0u;
        CRT_CUDA(cudaMemcpyAsync(keys, init, sizeof(init), cudaMemcpyHostToDevice, st));
        k_bounds<<<std::min<uint32_t>(cdiv(n, BLOCK), (uint32_t)ctx->sm_count * 4), BLOCK, 0, st>>>(tbox, cen, n, keys);
        check_launch(ctx, "k_bounds");
        k_morton<<<cdiv(n, BLOCK), BLOCK, 0, st>>>(cen, n, keys, code_a, idx_a);
        check_launch(ctx, "k_morton");
        if (sah) CRT_CUDA(cudaMemcpyAsync(code_prim, code_a, 4ull * n, cudaMemcpyDeviceToDevice, st));
        const uint32_t nb = cdiv(n, SORT_TILE);
        uint32_t *ka = code_a, *va = idx_a, *kb = code_b, *vb = idx_b;
        for (int shift = 0; shift < 32; shift += 8) {
            k_radix_hist<<<nb, SORT_THREADS, 0, st>>>(ka, n, shift, hist);
            check_launch(ctx, "k_radix_hist");
            k_scan<<<1, 1024, 0, st>>>(hist, nb * 256);
            check_launch(ctx, "k_scan");
            k_radix_scatter<<<nb, SORT_THREADS, 0, st>>>(ka, va, kb, vb, n, shift, hist);
            check_launch(ctx, "k_radix_scatter");
            std::swap(ka, kb);
            std::swap(va, vb);
        }
        // after 4 passes the sorted data is back in (code_a, idx_a)
        if (sah) {
            sah_topology(ctx, (int)n, sah_temp, tbox, cen, keys, va, code_prim, child, range, parent, root);
        } else if (n > 1) {
            k_karras<<<cdiv(n - 1, BLOCK), BLOCK, 0, st>>>(ka, (int)n, child, range, parent);
            check_launch(ctx, "k_karras");
        }
        if (ctx->treelet_passes > 0 && n >= 8) {
            // treelet restructuring of the binary tree, then leaves renumbered depth-first
            k_tl_boxes<<<cdiv(n, BLOCK), BLOCK, 0, st>>>(va, tbox, (int)n, child, parent, nbox, flags, ctx->d_error);
            check_launch(ctx, "k_tl_boxes");
            const uint32_t tl_grid = std::min<uint32_t>(cdiv(n - 1, TL_WARPS), (uint32_t)ctx->sm_count * 16);
            // root lists (tl_pos, filled later, has room) and their lengths, one per launch
            uint32_t* tl_count = keys + 32;
            for (uint32_t pass = 0; pass < ctx->treelet_passes; ++pass) {
                CRT_CUDA(cudaMemsetAsync(tl_count, 0, 7 * sizeof(uint32_t), st));
                for (int cls = 0; cls < 7; ++cls) {
                    k_tl_roots<<<cdiv(n - 1, BLOCK), BLOCK, 0, st>>>(parent, child, (int)n, cls, tl_pos, tl_count + cls);
                    check_launch(ctx, "k_tl_roots");
                    k_treelet<<<tl_grid, 32 * TL_WARPS, 0, st>>>(child, parent, nbox, tl_pos, tl_count + cls, (int)n);
                    check_launch(ctx, "k_treelet");
                }
            }
            CRT_CUDA(cudaMemsetAsync(flags, 0, nn * 4, st));
            k_tl_count<<<cdiv(n, BLOCK), BLOCK, 0, st>>>((int)n, child, parent, tl_cnt, flags, ctx->d_error);
            check_launch(ctx, "k_tl_count");
            k_tl_position<<<cdiv(2 * n - 1, BLOCK), BLOCK, 0, st>>>((int)n, child, parent, tl_cnt, tl_pos,
                                                                   ctx->d_error);
            check_launch(ctx, "k_tl_position");
            k_tl_relayout<<<cdiv(n, BLOCK), BLOCK, 0, st>>>((int)n, tl_pos, tl_cnt, va, tl_sorted, child, range, parent,
                                                           tl_par, ctx->d_error);
            check_launch(ctx, "k_tl_relayout");
            CRT_CUDA(cudaMemcpyAsync(va, tl_sorted, 4ull * n, cudaMemcpyDeviceToDevice, st));
            CRT_CUDA(cudaMemcpyAsync(parent + (n - 1), tl_par, 4ull * n, cudaMemcpyDeviceToDevice, st));
            CRT_CUDA(cudaMemsetAsync(flags, 0, nn * 4, st));
        }
        k_refit<<<cdiv(n, BLOCK), BLOCK, 0, st>>>(va, tbox, (int)n, child, parent, nbox, flags, range, dpc,
                                                  ctx->collapse_tri_cost, ctx->d_error);
        check_launch(ctx, "k_refit");
        idx_a = va;
    }

    CRT_CUDA(cudaMalloc(&s->tris, sizeof(float4) * 3 * nn));
    CRT_CUDA(cudaMalloc(&s->leaf_prim, sizeof(uint32_t) * nn));
    CRT_CUDA(cudaMalloc(&s->leaf_entity, sizeof(uint32_t) * nn));
    if (any_vn) CRT_CUDA(cudaMalloc(&s->leaf_vn, sizeof(float4) * 3 * nn));
    const int2 whole = make_int2(n > 3 ? 0 : ALL_TRIS, 0);
    if (sah) CRT_CUDA(cudaMemsetAsync(&root->y, 0, sizeof(int), st));
    else CRT_CUDA(cudaMemcpyAsync(root, &whole, sizeof(whole), cudaMemcpyHostToDevice, st));

    CollapseArgs A;
    A.n = (int)n;
    A.child = child;
    A.range = range;
    A.nbox = nbox;
    A.sorted = idx_a;
    A.geo = geo;
    A.vn = any_vn ? vn : nullptr;
    A.prim_ent = prim_ent;
    A.tris = s->tris;
    A.leaf_prim = s->leaf_prim;
    A.leaf_vn = s->leaf_vn;
    A.leaf_entity = s->leaf_entity;
    A.counters = counts;
    A.err = ctx->d_error;
    A.dp = dpc;
    A.cost_tri = ctx->collapse_tri_cost;

    // Wide-node capacity.  Every wide node but the root holds more than three triangles, and a tree that
    // fills its nodes has fewer than n / 3.  That is no bound: where all costs are equal (a body whose FP32
    // vertices coincide, far from the origin: every area zero) or lost beside a much larger one, nodes stay whole
    // with two children each.  Such a collapse runs out of nodes, counts on (used[0]) and is done again
    // with a node for every internal node of the binary tree, the most there can be.
    uint32_t cap = std::max<uint32_t>(1, n / 3 + 2), depth = 0;
    uint32_t used[2 + COLLAPSE_MAX_LEVELS + 1];   // nodes, triangles, nodes per level
    const uint32_t* const per_level = used + 2;
    for (;;) {
        CRT_CUDA(cudaMalloc(&s->nodes, sizeof(WideNode) * cap));
        A.nodes = s->nodes;
        A.node_cap = cap;
        const uint32_t c0[3] = {1, 0, 1};
        CRT_CUDA(cudaMemsetAsync(counts, 0, sizeof(used), st));
        CRT_CUDA(cudaMemcpyAsync(counts, c0, sizeof(c0), cudaMemcpyHostToDevice, st));
        // The levels are launched without waiting for their sizes, which stay on the device (level d of the
        // tree has at most 8^d nodes): as many as a tree of this size usually has, then a look at the counts,
        // then two at a time.
        const int2* cur = root;
        int2* nxt = front;
        uint32_t launched = 0, batch = 4;
        for (uint32_t m = n / 3; m; m /= 8) ++batch;
        for (uint64_t bound = 1;;) {
            CRT_CHECK(launched + batch <= COLLAPSE_MAX_LEVELS, CRT_ERR_DEVICE, "BVH collapse did not terminate");
            for (uint32_t b = 0; b < batch; ++b, ++launched) {
                const uint32_t grid = std::min<uint32_t>(cdiv(bound, COLLAPSE_BLOCK / 8), (uint32_t)ctx->sm_count * 16);
                k_collapse<<<grid, COLLAPSE_BLOCK, 0, st>>>(A, cur, counts + 2 + launched, nxt);
                check_launch(ctx, "k_collapse");
                cur = nxt;
                nxt = nxt == front ? front_b : front;
                bound = std::min<uint64_t>(bound * 8, cap);
            }
            CRT_CUDA(cudaMemcpyAsync(used, counts, sizeof(uint32_t) * (2 + launched + 1), cudaMemcpyDeviceToHost, st));
            CRT_CUDA(cudaStreamSynchronize(st));
            if (!per_level[launched]) break;
            batch = 2;
        }
        for (depth = 0; depth < launched && per_level[depth];) ++depth;
        if (used[0] <= cap) break;
        CRT_CHECK(cap < n, CRT_ERR_DEVICE, "BVH collapse has more nodes than its binary tree");
        CRT_CUDA(cudaFree(s->nodes));
        s->nodes = nullptr;
        cap = n;
    }
    uint32_t kb_h[6] = {0, 0, 0, 0, 0, 0};
    if (n) CRT_CUDA(cudaMemcpyAsync(kb_h, keys, sizeof(kb_h), cudaMemcpyDeviceToHost, st));
    CRT_CUDA(cudaEventRecord(ev1, st));
    CRT_CUDA(cudaStreamSynchronize(st));
    check_device_error(ctx, "BVH build");
    CRT_CHECK(used[1] == n, CRT_ERR_DEVICE, "BVH collapse placed " + std::to_string(used[1]) + " of " +
                                                std::to_string(n) + " triangles");
    float ms = 0;
    CRT_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    s->build_ms = ms;
    s->n_nodes = used[0];
    s->depth = depth;
    // the node array was sized for the worst case (n / 3 + 2 nodes); keep only the nodes used
    if (used[0] < cap) {
        WideNode* exact = nullptr;
        CRT_CUDA(cudaMalloc(&exact, sizeof(WideNode) * std::max<uint32_t>(used[0], 1)));
        CRT_CUDA(cudaMemcpyAsync(exact, s->nodes, sizeof(WideNode) * used[0], cudaMemcpyDeviceToDevice, st));
        CRT_CUDA(cudaStreamSynchronize(st));
        CRT_CUDA(cudaFree(s->nodes));
        s->nodes = exact;
    }
    for (int k = 0; k < 6; ++k) s->bounds[k] = n ? fkey_inv(kb_h[k]) : 0.f;
    s->device_bytes = sizeof(WideNode) * std::max<uint32_t>(used[0], 1) + nn * (48 + 4 + 4) + (any_vn ? nn * 48 : 0) +
                      sizeof(EntityDev) * s->host_entities.size();
}
