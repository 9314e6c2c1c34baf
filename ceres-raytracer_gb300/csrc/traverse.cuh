// Traversal of the 8-wide compressed BVH (device code).
//
// Semantics follow SingleRayTraverser (lib/bvh/single_ray_traverser.hpp:68-126) with
// Closest/AnyPrimitiveIntersector: every triangle whose test passes shrinks tmax (closest hit) or
// ends the traversal (any hit).  Leaves are intersected as soon as their parent node is visited
// (the reference's "eager" leaves); internal children are visited nearest-first by the octant
// order fixed at build time.  Node groups (base index, hit bits, slot mask) live on a per-thread
// stack whose first STACK_SMEM entries are in shared memory and the rest in local memory.  The
// triangle test is watertight (tri_test); the child-box test reads the node's planes two to a word
// (WideNode), and the ray octant picks each axis's entry / exit row by address.
//
// What bounds it: instruction issue (and, for incoherent rays, the L1 data pipe and its latency).  The
// node test is therefore written for few instructions: half of the planes need no decoding, two planes
// take one packed fma, a child's hit is one sign bit shifted into a mask, and the triangles of all leaf
// children that were hit come from that mask by four multiplies and masks.  Against planes as halves
// with one conversion and one fma each, and a byte of slot / triangle bits looked up per child: 18 - 23 %
// fewer instructions, and the kernel then waits for memory more than for issue slots (0.60 -> 0.53 of a
// slot used per cycle on incoherent rays), so it runs as many warps as it can (8 blocks per SM, below).
// Together, before / after: 3 M incoherent closest-hit rays on 2 M triangles 1942 / 1742 us, 333 k any-hit
// rays on 100 k 125 / 120 us, a 1024^2 beam scan 236 / 211 us, a 2048^2 render 1860 / 1625 us, 12 x 2048^2
// sun rays 3260 / 3070 us.  (Times of one workload differ between comments with the body's pose and the timing
// loop; a pair is of one pose.)
#pragma once

#include "common.cuh"
#include <cuda_fp16.h>

#ifndef CRT_STACK_SMEM
#define CRT_STACK_SMEM 8
#endif
#ifndef CRT_TRACE_BLOCK
#define CRT_TRACE_BLOCK 128   // threads of a trace block (the strides of its shared memory)
#endif
#define CRT_STACK_TOTAL 64   // > wide-tree depth bound (binary depth <= 62 with index tie-breaks)

struct SceneView {
    const WideNode* __restrict__ nodes;
    const float4* __restrict__ tris;
    const uint32_t* __restrict__ leaf_prim;
    const float4* __restrict__ leaf_vn;
    const uint32_t* __restrict__ leaf_entity;
    const EntityDev* __restrict__ entities;
    uint32_t n_tris;
};

struct TravStats {
    uint32_t nodes, tris;
};

// Shared memory of a trace block, every array indexed by thread last (no bank conflicts): the first
// stack entries (8 bytes each), four float4 of ray constants that only the triangle test reads, and one
// float4 of the closest hit so far.  Keeping those 18 values out of the registers while nodes are
// visited is what brings the kernels to 8 blocks per SM (64 registers) with little or no spilling; a
// triangle group reads them back with four 16-byte loads.  (In registers, the beam scan's kernel spilled
// even at 7 blocks: 243 us against 211.)
constexpr uint32_t TRACE_RAY = 8u * CRT_STACK_SMEM * CRT_TRACE_BLOCK;   // byte offsets
constexpr uint32_t TRACE_ROW = 16u * CRT_TRACE_BLOCK;
constexpr uint32_t TRACE_HIT = TRACE_RAY + 4u * TRACE_ROW;
constexpr uint32_t TRACE_SMEM = TRACE_HIT + TRACE_ROW;

// volatile: the values are to live in shared memory, not in registers
__device__ __forceinline__ void st_shared4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ float4 ld_shared4(uint32_t a) {
    float4 r;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                 : "r"(a)
                 : "memory");
    return r;
}

// A pair of floats in one 64-bit register pair, and fma of both in one instruction (fma.rn.f32x2): each
// lane's result is that of fmaf.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The planes of two neighbouring words of a row (WideNode): of the even children as the words are, of
// the odd ones from the words' low halves, whose sign bit belongs to the even child.
__device__ __forceinline__ f32x2 planes(float w0, float w1, bool odd) {
    if (!odd) return pack2(w0, w1);
    const __half h0 = __ushort_as_half((unsigned short)(__float_as_uint(w0) & 0xFFFFu));
    const __half h1 = __ushort_as_half((unsigned short)(__float_as_uint(w1) & 0xFFFFu));
    return pack2(__half2float(__habs(h0)), __half2float(__habs(h1)));
}

// The end of a ray's range, and with it the distance of a hit, is never -0: a child whose exit is -0 and whose
// entry +0 would count as missed (visits below), although the triangle test takes them for equal.
__device__ __forceinline__ float not_neg0(float t) { return __fadd_rn(t, 0.0f); }

// What a node visit needs of the ray.
struct NodeRay {
    float3 idir, ood;
    uint32_t rowx, rowy, rowz;      // rows of the entry planes per axis (lo rows 2..4, hi rows 5..7; a negative
                                    // direction enters at hi), as byte offsets; the exit row is the entry row's
                                    // partner, an exclusive or away
    uint32_t pick2, pick1, pick0;   // per slot bit, the slots that differ from the octant in it (in the group's top byte)
};
__device__ __forceinline__ NodeRay node_ray(const TRay& ray) {
    // octant from the sign bits, as NodeIntersector does with std::signbit (node_intersectors.hpp:25-30):
    // -0.0 counts as negative, consistent with safe_rcp(-0.0) < 0
    const uint32_t oct = (__float_as_uint(ray.d.x) >> 31) | ((__float_as_uint(ray.d.y) >> 31) << 1) |
                         ((__float_as_uint(ray.d.z) >> 31) << 2);
    NodeRay c;
    c.idir = f3(safe_rcp(ray.d.x), safe_rcp(ray.d.y), safe_rcp(ray.d.z));
    c.ood = f3(-ray.o.x * c.idir.x, -ray.o.y * c.idir.y, -ray.o.z * c.idir.z);
    c.rowx = (oct & 1u) ? 0x50u : 0x20u;
    c.rowy = (oct & 2u) ? 0x60u : 0x30u;
    c.rowz = (oct & 4u) ? 0x70u : 0x40u;
    c.pick2 = (oct & 4u) ? 0x0F000000u : 0xF0000000u;
    c.pick1 = (oct & 2u) ? 0x33000000u : 0xCC000000u;
    c.pick0 = (oct & 1u) ? 0x55000000u : 0xAA000000u;
    return c;
}

// Takes the internal child to visit next out of a group and returns its node: the pending one whose slot
// differs most from the octant.
__device__ __forceinline__ uint32_t next_child(uint2& group, const NodeRay& c) {
    uint32_t cb = group.y & 0xFF000000u;   // pending children; ends as the one taken
    uint32_t pr = cb & c.pick2;
    cb = pr ? pr : cb;
    pr = cb & c.pick1;
    cb = pr ? pr : cb;
    pr = cb & c.pick0;
    cb = pr ? pr : cb;
    const uint32_t node = group.x + __popc(group.y & ((cb >> 24) - 1u));
    group.y ^= cb;
    return node;
}

// Each child's bit spread to three, one per triangle of a leaf (ascending bits are ascending slots).
__device__ __forceinline__ uint32_t leaf_bits(uint32_t hits) {
    uint32_t leaf3 = hits & 0xFFu;
    leaf3 = (leaf3 * 0x101u) & 0x00F00Fu;
    leaf3 = (leaf3 * 0x11u) & 0x0C30C3u;
    leaf3 = (leaf3 * 0x5u) & 0x249249u;
    return leaf3 * 7u;
}

// Tests the 8 quantised child boxes of a node: the group of internal children that the ray meets, and the
// triangles of the leaf children that it meets (tmask, of the node's tvalid, from tbase on).
__device__ __forceinline__ void visit_node(const WideNode* __restrict__ nodes, uint32_t node, const NodeRay& c, float tmin,
                                           float tmax, uint2& group, uint32_t& tmask, uint32_t& tvalid, uint32_t& tbase) {
    const uintptr_t np = reinterpret_cast<uintptr_t>(nodes + node) ^ ((node & 7u) << 4);   // rows permuted
    auto row = [&](uint32_t off) { return __ldg(reinterpret_cast<const float4*>(np ^ off)); };
    const float4 w0 = row(0x00u), w1 = row(0x10u);
    const uint32_t ew = __float_as_uint(w0.w);
    const float sx = __uint_as_float(ew & 0x7F800000u) * c.idir.x;
    const float sy = __uint_as_float((ew << 8) & 0x7F800000u) * c.idir.y;
    const float sz = __uint_as_float((ew << 16) & 0x7F800000u) * c.idir.z;
    const float ax = fmaf(-256.0f, sx, fmaf(w0.x, c.idir.x, c.ood.x));
    const float ay = fmaf(-256.0f, sy, fmaf(w0.y, c.idir.y, c.ood.y));
    const float az = fmaf(-256.0f, sz, fmaf(w0.z, c.idir.z, c.ood.z));
    const f32x2 sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
    const f32x2 ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
    // entry / exit planes per axis by the ray octant: the lo / hi rows swap by address
    const float4 xn = row(c.rowx), xf = row(c.rowx ^ 0x70u), yn = row(c.rowy), yf = row(c.rowy ^ 0x50u), zn = row(c.rowz),
                 zf = row(c.rowz ^ 0x30u);
    // exit minus entry distance of each child: its sign bit is set where the ray misses the child
    // (the difference of two floats is zero only where they are equal).  Children 7 .. 0 are shifted
    // into `miss` in turn.
    uint32_t miss = 0;
#pragma unroll
    for (int half = 1; half >= 0; --half) {   // children 4 half .. 4 half + 3: two words of each row
        float2 gap[2];
#pragma unroll
        for (int odd = 1; odd >= 0; --odd) {
            auto dist = [&](const float4& r, f32x2 s, f32x2 a) {
                return unpack2(fma2(half ? planes(r.z, r.w, odd) : planes(r.x, r.y, odd), s, a));
            };
            const float2 tx0 = dist(xn, sx2, ax2), tx1 = dist(xf, sx2, ax2);
            const float2 ty0 = dist(yn, sy2, ay2), ty1 = dist(yf, sy2, ay2);
            const float2 tz0 = dist(zn, sz2, az2), tz1 = dist(zf, sz2, az2);
            gap[odd].x = fminf(fminf(tx1.x, ty1.x), fminf(tz1.x, tmax)) -
                         fmaxf(fmaxf(tx0.x, ty0.x), fmaxf(tz0.x, tmin));
            gap[odd].y = fminf(fminf(tx1.y, ty1.y), fminf(tz1.y, tmax)) -
                         fmaxf(fmaxf(tx0.y, ty0.y), fmaxf(tz0.y, tmin));
        }
        miss = __funnelshift_l(__float_as_uint(gap[1].y), miss, 1);
        miss = __funnelshift_l(__float_as_uint(gap[0].y), miss, 1);
        miss = __funnelshift_l(__float_as_uint(gap[1].x), miss, 1);
        miss = __funnelshift_l(__float_as_uint(gap[0].x), miss, 1);
    }
    const uint32_t vm = __float_as_uint(w1.z);   // 24 bits of triangles, 8 of internal children
    const uint32_t hits = ~miss;
    tvalid = vm & 0x00FFFFFFu;
    tmask = leaf_bits(hits) & tvalid;
    tbase = __float_as_uint(w1.y);
    group = make_uint2(__float_as_uint(w1.x), ((hits << 24) & vm) | (vm >> 24));
}

// The ray constants of the triangle test, and no hit, into the lane's place.
template <bool ANY>
__device__ __forceinline__ void ray_to_shared(const TRay& ray, uint32_t own) {
    const TShear sh = make_shear(ray.d);
    st_shared4(own + TRACE_RAY, sh.bx.x, sh.bx.y, sh.bx.z, shear_proj(ray.o, sh.bx));
    st_shared4(own + TRACE_RAY + TRACE_ROW, sh.by.x, sh.by.y, sh.by.z, shear_proj(ray.o, sh.by));
    st_shared4(own + TRACE_RAY + 2 * TRACE_ROW, ray.o.x, ray.o.y, ray.o.z, __uint_as_float(ray.skip));
    st_shared4(own + TRACE_RAY + 3 * TRACE_ROW, ray.d.x, ray.d.y, ray.d.z, ray.tmin);
    if (!ANY) st_shared4(own + TRACE_HIT, 0.f, 0.f, 1.f, __uint_as_float(CRT_MISS));
}

// smem: the block's TRACE_SMEM bytes.  An any-hit traversal returns the slot only.
template <bool ANY, bool COUNT>
__device__ __forceinline__ THit traverse(const SceneView& sv, TRay ray, unsigned char* smem, TravStats& st,
                                         uint32_t* __restrict__ err) {
    THit hit;
    hit.slot = CRT_MISS;
    hit.t = hit.u = hit.v = 0.f;
    ray.tmax = not_neg0(ray.tmax);
    uint2* const sstack = reinterpret_cast<uint2*>(smem) + threadIdx.x;
    const uint32_t own = (uint32_t)__cvta_generic_to_shared(smem) + 16u * threadIdx.x;
    const NodeRay nr = node_ray(ray);
    ray_to_shared<ANY>(ray, own);
    uint2 lstack[CRT_STACK_TOTAL - CRT_STACK_SMEM];
    int sp = 0;
    // root = slot 0 of a virtual parent whose children start at node 0
    uint2 ngroup = make_uint2(0u, 0x01000001u);
    uint32_t tmask = 0, tvalid = 0, tbase = 0;
    while (true) {
        // ---- leaf triangles of the last visited node
        if (tmask) {
            TRay r;
            TShear shear;
            const float4 q0 = ld_shared4(own + TRACE_RAY), q1 = ld_shared4(own + TRACE_RAY + TRACE_ROW);
            const float4 q2 = ld_shared4(own + TRACE_RAY + 2 * TRACE_ROW), q3 = ld_shared4(own + TRACE_RAY + 3 * TRACE_ROW);
            shear.bx = f3(q0.x, q0.y, q0.z);
            shear.ox = q0.w;
            shear.by = f3(q1.x, q1.y, q1.z);
            shear.oy = q1.w;
            r.o = f3(q2.x, q2.y, q2.z);
            r.skip = __float_as_uint(q2.w);
            r.d = f3(q3.x, q3.y, q3.z);
            r.tmin = q3.w;
            do {
                const uint32_t low = tmask & (0u - tmask);
                tmask ^= low;
                const uint32_t slot = tbase + __popc(tvalid & (low - 1u));
                if (slot == r.skip) continue;
                const float4* tp = sv.tris + 3ull * slot;
                const float4 a = __ldg(tp), bb = __ldg(tp + 1), c = __ldg(tp + 2);
                if (COUNT) st.tris++;
                r.tmax = ray.tmax;
                float t, wv, ww, det;
                if (tri_test(a, bb, c, r, shear, t, wv, ww, det)) {
                    if (ANY) {
                        hit.slot = slot;
                        return hit;
                    }
                    ray.tmax = not_neg0(t);
                    st_shared4(own + TRACE_HIT, wv, ww, det, __uint_as_float(slot));
                }
            } while (tmask);
        }
        // ---- next internal node
        if (ngroup.y <= 0x00FFFFFFu) {
            if (sp == 0) break;
            --sp;
            ngroup = sp < CRT_STACK_SMEM ? sstack[sp * CRT_TRACE_BLOCK] : lstack[sp - CRT_STACK_SMEM];
        }
        const uint32_t node = next_child(ngroup, nr);
        if (ngroup.y > 0x00FFFFFFu) {
            if (sp < CRT_STACK_SMEM) sstack[sp * CRT_TRACE_BLOCK] = ngroup;
            else if (sp < CRT_STACK_TOTAL) lstack[sp - CRT_STACK_SMEM] = ngroup;
            else {
                atomicOr(err, (uint32_t)DEVERR_STACK_OVERFLOW);
                break;
            }
            ++sp;
        }
        if (COUNT) st.nodes++;
        visit_node(sv.nodes, node, nr, ray.tmin, ray.tmax, ngroup, tmask, tvalid, tbase);
    }
    if (ANY) return hit;
    const float4 h = ld_shared4(own + TRACE_HIT);   // weights of p1 and p2, their sum with p0's, slot
    hit.slot = __float_as_uint(h.w);
    const float inv = 1.0f / h.z;
    hit.t = hit.slot != CRT_MISS ? ray.tmax : 0.0f;
    hit.u = h.x * inv;
    hit.v = h.y * inv;
    return hit;
}

// ---------------------------------------------------------------- triangles dealt to the warp
// The same traversal for incoherent rays.  After a node a few lanes of such a warp have several triangles
// each and the others none; tested by their own lanes they take as many rounds of the triangle test as
// the lane with the most has.  Here the warp steps together, and when few triangles are spread unevenly
// they are dealt to the lanes, 32 a round, which read the owner's ray from shared memory and report a hit
// there.  The nodes visited and the hits are those of traverse (of equal distances the last triangle wins).
// Lanes that step together wait for each other, and on coherent rays that costs more than dealing gives:
// 2048^2 camera rays in tiles take 10 - 15 % longer this way, so it is for rays that are likely to be
// incoherent (trace_coop).  Per kernel and without it: 3 M random closest-hit rays on 2 M triangles 1500 /
// 1350 us, 333 k any-hit rays on 100 k 101 / 93 us; with the bounce, later shadow and specular rays of a
// 24-image batch 3530 / 3466 us, of 12 x 2048^2 sun rays 2645 / 2592 us (whole calls).
// rays_apart: whether the rays of a warp are such: their directions are of several octants, or their
// origins lie further apart than an eighth of the scene.  For buffers of rays, of which nothing is known:
// with it 2048^2 camera rays in tiles take 3 - 6 % longer than in a kernel with traverse alone, against the 10
// - 15 % (closest hits on 20 k / 500 k / 2 M triangles: 303 / 387 / 436 us alone, 314 / 399 / 449 with
// both; any hits 213 / 272 / 329 and 228 / 288 / 347).  Least is gained just above SMALL_SCENE: 45 k rays on
// 1,100 triangles without / with both, random 28.7 / 26.9 us, coherent 21.9 / 23.1.
__device__ __forceinline__ bool rays_apart(const SceneView& sv, const TRay& ray, bool active) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    const uint32_t live = __ballot_sync(ALL, active);
    if (!live) return false;
    const int first = __ffs(live) - 1;
    const uint32_t ew = __float_as_uint(__ldg(reinterpret_cast<const float4*>(sv.nodes)).w);
    const float step = fmaxf(fmaxf(__uint_as_float(ew & 0x7F800000u), __uint_as_float((ew << 8) & 0x7F800000u)),
                             __uint_as_float((ew << 16) & 0x7F800000u));   // the scene is at most 256 of these wide
    const float dx = fabsf(ray.o.x - __shfl_sync(ALL, ray.o.x, first)), dy = fabsf(ray.o.y - __shfl_sync(ALL, ray.o.y, first)),
                dz = fabsf(ray.o.z - __shfl_sync(ALL, ray.o.z, first));
    const uint32_t turn = (__float_as_uint(ray.d.x) ^ __float_as_uint(__shfl_sync(ALL, ray.d.x, first))) |
                          (__float_as_uint(ray.d.y) ^ __float_as_uint(__shfl_sync(ALL, ray.d.y, first))) |
                          (__float_as_uint(ray.d.z) ^ __float_as_uint(__shfl_sync(ALL, ray.d.z, first)));
    const bool apart = (turn >> 31) || fmaxf(fmaxf(dx, dy), dz) > 32.0f * step;
    return __any_sync(ALL, active && apart);
}

// smem: the block's COOP_SMEM bytes.  An any-hit traversal returns a slot of 0 for a hit.  Called by the
// whole warp; `active`: the lane has a ray.
constexpr uint32_t COOP_OWNER = TRACE_SMEM;   // a lane number per thread
constexpr uint32_t COOP_SMEM = COOP_OWNER + CRT_TRACE_BLOCK;
template <bool ANY, bool COUNT>
__device__ __forceinline__ THit traverse_coop(const SceneView& sv, TRay ray, bool active, unsigned char* smem,
                                              TravStats& st, uint32_t* __restrict__ err) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    THit hit;
    hit.slot = CRT_MISS;
    hit.t = hit.u = hit.v = 0.f;
    ray.tmax = not_neg0(ray.tmax);
    uint2* const sstack = reinterpret_cast<uint2*>(smem) + threadIdx.x;
    const uint32_t own = (uint32_t)__cvta_generic_to_shared(smem) + 16u * threadIdx.x;
    const NodeRay nr = node_ray(ray);
    ray_to_shared<ANY>(ray, own);
    // the nearest hit of a round is found in the first half of the owner's hit row
    auto best = [&](uint32_t thread) { return reinterpret_cast<unsigned long long*>(smem + TRACE_HIT + 16u * thread); };
    uint8_t* const s_owner = smem + COOP_OWNER + (threadIdx.x & ~31u);
    uint2 lstack[CRT_STACK_TOTAL - CRT_STACK_SMEM];
    int sp = 0;
    // root = slot 0 of a virtual parent whose children start at node 0
    uint2 ngroup = make_uint2(0u, active ? 0x01000001u : 0u);
    uint32_t tmask = 0, tvalid = 0, tbase = 0;
    while (true) {
        // ---- leaf triangles of the last visited node
        const bool with = __any_sync(ALL, tmask != 0u);
        bool deal = false;
        if (with) {
            // A round of dealt triangles takes about as long as 1.6 of the lanes' own, plus 0.6 to deal.
            // (Dealing whenever a lane has three or more, 12 x 2048^2 sun rays take 6 % longer and
            // small mirror-like scenes up to 1.6 times; only with at most 16 or 8 lanes that have
            // triangles, 3 M random rays take 0.3 % and 2.4 % longer.)
            const uint32_t own_rounds = __reduce_max_sync(ALL, (uint32_t)__popc(tmask));
            const uint32_t sum = __reduce_add_sync(ALL, (uint32_t)__popc(tmask));
            deal = 5u * own_rounds > 3u + 8u * ((sum + 31u) >> 5);
        }
        if (deal) {
            // the warp's triangles dealt to its lanes, 32 at a time
            const uint32_t lane = threadIdx.x & 31u;
            const uint32_t cnt = __popc(tmask);
            uint32_t incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(ALL, incl, o);
                if ((int)lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(ALL, incl, 31), first = incl - cnt;
            bool found = false;
            for (uint32_t r0 = 0; r0 < total; r0 += 32u) {
                // owners with triangles among [r0, r0 + 32): one bit at each one's first place
                const bool here = cnt && incl > r0 && first < r0 + 32u;
                const uint32_t place = max(first, r0) - r0;
                const uint32_t starts = __reduce_or_sync(ALL, here ? 1u << place : 0u);
                const uint32_t owners = __ballot_sync(ALL, here);
                const uint32_t upto = starts & (0xFFFFFFFFu >> (31u - lane));
                if (here) s_owner[__popc(owners & ((1u << lane) - 1u))] = (uint8_t)lane;
                __syncwarp();
                const uint32_t o = s_owner[__popc(upto) - 1];   // the lane's owner
                const uint32_t ofirst = __shfl_sync(ALL, first, o), ocnt = __shfl_sync(ALL, cnt, o);
                uint32_t m = __shfl_sync(ALL, tmask, o);
                const uint32_t ovalid = __shfl_sync(ALL, tvalid, o), obase = __shfl_sync(ALL, tbase, o);
                const float otmax = __shfl_sync(ALL, ray.tmax, o);
                const float4* const otris = reinterpret_cast<const float4*>(__shfl_sync(ALL, reinterpret_cast<unsigned long long>(sv.tris), o));
                const uint32_t k = r0 + lane - ofirst;
                bool ok = false;
                float t = 0.f, wv = 0.f, ww = 0.f, det = 1.f;
                uint32_t slot = 0;
                const uint32_t ow = own + 16u * (o - lane);
                if (r0 + lane < total && k < ocnt) {
                    for (uint32_t q = 0; q < k; ++q) m &= m - 1u;
                    slot = obase + __popc(ovalid & ((m & (0u - m)) - 1u));
                    TRay r;
                    TShear shear;
                    const float4 q2 = ld_shared4(ow + TRACE_RAY + 2 * TRACE_ROW);
                    r.o = f3(q2.x, q2.y, q2.z);
                    r.skip = __float_as_uint(q2.w);
                    if (slot != r.skip) {
                        const float4* tp = otris + 3ull * slot;
                        const float4 a = __ldg(tp), bb = __ldg(tp + 1), c = __ldg(tp + 2);
                        const float4 q0 = ld_shared4(ow + TRACE_RAY), q1 = ld_shared4(ow + TRACE_RAY + TRACE_ROW);
                        const float4 q3 = ld_shared4(ow + TRACE_RAY + 3 * TRACE_ROW);
                        shear.bx = f3(q0.x, q0.y, q0.z);
                        shear.ox = q0.w;
                        shear.by = f3(q1.x, q1.y, q1.z);
                        shear.oy = q1.w;
                        r.d = f3(q3.x, q3.y, q3.z);
                        r.tmin = q3.w;
                        r.tmax = otmax;
                        if (COUNT) st.tris++;
                        ok = tri_test(a, bb, c, r, shear, t, wv, ww, det);
                    }
                }
                const uint32_t hits = __reduce_or_sync(ALL, ok ? 1u << o : 0u);
                if (hits) {
                    const bool mine = (hits >> lane) & 1u;
                    if (ANY) {
                        found = found || mine;
                    } else {
                        // per owner the nearest, of equal ones the last: as when they are tested in turn
                        const uint32_t tu = __float_as_uint(not_neg0(t));
                        const unsigned long long key = (unsigned long long)((tu & 0x80000000u) ? ~tu : (tu | 0x80000000u)) << 32 | (0xFFFFFFFFu - slot);
                        unsigned long long* const sb = best(threadIdx.x - lane + o);
                        if (mine) *best(threadIdx.x) = ~0ull;   // (the hit that was there is further away)
                        __syncwarp();
                        if (ok) atomicMin(sb, key);
                        __syncwarp();
                        const bool won = ok && *reinterpret_cast<volatile unsigned long long*>(sb) == key;
                        if (mine) {
                            const uint32_t u = (uint32_t)(*reinterpret_cast<volatile unsigned long long*>(best(threadIdx.x)) >> 32);
                            ray.tmax = __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
                        }
                        __syncwarp();
                        if (won) st_shared4(ow + TRACE_HIT, wv, ww, det, __uint_as_float(slot));
                        __syncwarp();
                    }
                }
            }
            if (ANY && found) {
                hit.slot = 0;
                ngroup.y = 0;
                sp = 0;
            }
            tmask = 0;
        } else if (with) {
            bool stop = false;
            if (tmask) {
                TRay r;
                TShear shear;
                const float4 q0 = ld_shared4(own + TRACE_RAY), q1 = ld_shared4(own + TRACE_RAY + TRACE_ROW);
                const float4 q2 = ld_shared4(own + TRACE_RAY + 2 * TRACE_ROW), q3 = ld_shared4(own + TRACE_RAY + 3 * TRACE_ROW);
                shear.bx = f3(q0.x, q0.y, q0.z);
                shear.ox = q0.w;
                shear.by = f3(q1.x, q1.y, q1.z);
                shear.oy = q1.w;
                r.o = f3(q2.x, q2.y, q2.z);
                r.skip = __float_as_uint(q2.w);
                r.d = f3(q3.x, q3.y, q3.z);
                r.tmin = q3.w;
                do {
                    const uint32_t low = tmask & (0u - tmask);
                    tmask ^= low;
                    const uint32_t slot = tbase + __popc(tvalid & (low - 1u));
                    if (slot == r.skip) continue;
                    const float4* tp = sv.tris + 3ull * slot;
                    const float4 a = __ldg(tp), bb = __ldg(tp + 1), c = __ldg(tp + 2);
                    if (COUNT) st.tris++;
                    r.tmax = ray.tmax;
                    float t, wv, ww, det;
                    if (tri_test(a, bb, c, r, shear, t, wv, ww, det)) {
                        if (ANY) {
                            stop = true;
                            break;
                        }
                        ray.tmax = not_neg0(t);
                        st_shared4(own + TRACE_HIT, wv, ww, det, __uint_as_float(slot));
                    }
                } while (tmask);
            }
            if (ANY && stop) {
                hit.slot = 0;
                ngroup.y = 0;
                tmask = 0;
                sp = 0;
            }
        }
        // ---- next internal node
        bool go = ngroup.y > 0x00FFFFFFu;
        if (!go && sp != 0) {
            --sp;
            ngroup = sp < CRT_STACK_SMEM ? sstack[sp * CRT_TRACE_BLOCK] : lstack[sp - CRT_STACK_SMEM];
            go = true;
        }
        if (!__any_sync(ALL, go)) break;
        tmask = 0;
        if (go) {
            const uint32_t node = next_child(ngroup, nr);
            if (ngroup.y > 0x00FFFFFFu) {
                if (sp < CRT_STACK_SMEM) sstack[sp * CRT_TRACE_BLOCK] = ngroup;
                else if (sp < CRT_STACK_TOTAL) lstack[sp - CRT_STACK_SMEM] = ngroup;
                else {
                    // reported, so the call fails; the ray goes on without what its stack held (to end it here takes
                    // a check after every visit, 0.4 - 0.9 % of 333 k any-hit rays)
                    atomicOr(err, (uint32_t)DEVERR_STACK_OVERFLOW);
                    sp = -1;
                }
                ++sp;
            }
            if (COUNT) st.nodes++;
            visit_node(sv.nodes, node, nr, ray.tmin, ray.tmax, ngroup, tmask, tvalid, tbase);
        }
    }
    if (ANY) return hit;
    const float4 h = ld_shared4(own + TRACE_HIT);   // weights of p1 and p2, their sum with p0's, slot
    hit.slot = __float_as_uint(h.w);
    const float inv = 1.0f / h.z;
    hit.t = hit.slot != CRT_MISS ? ray.tmax : 0.0f;
    hit.u = h.x * inv;
    hit.v = h.y * inv;
    return hit;
}

// ---------------------------------------------------------------- eight lanes per ray
// The same traversal for launches of few rays, which last as long as their longest chain of dependent
// node visits: lane c of a ray's eight lanes tests child c, and up to eight triangles are tested at once.
// The four rays of a warp step together.  Visits, hits and their order are those of traverse: of the
// triangles of one step the nearest wins, of equal ones the last, as when they are tested in turn.
// What bounds it is the length of one step: the loads of a node (a word per plane and lane), a child's slab
// test, the choice of the next child, the loads and test of its triangles.  Against a lane per ray, in
// groups small enough to fill the GPU: 256 rays on 20 k triangles 22.4 -> 16.8 us, a 128^2 render 125 ->
// 93 us, a 250^2 sun-ray grid with two bounces 130 -> 113 us.
constexpr uint32_t OCT_RAYS = CRT_TRACE_BLOCK / 8;                        // rays of a block
constexpr uint32_t OCT_SMEM = 8u * CRT_STACK_TOTAL * OCT_RAYS;   // their stacks, indexed by ray last

// Called by the whole warp; `active`, the ray and the scene are the same for a ray's eight lanes.
template <bool ANY, bool COUNT>
__device__ __forceinline__ THit traverse_oct(const SceneView& sv, TRay ray, bool active, unsigned char* smem,
                                             TravStats& st, uint32_t* __restrict__ err) {
    constexpr uint32_t ALL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, oct0 = lane & 24u;
    THit hit;
    hit.slot = CRT_MISS;
    hit.t = hit.u = hit.v = 0.f;
    ray.tmax = not_neg0(ray.tmax);
    float det = 1.0f;
    uint2* const stack = reinterpret_cast<uint2*>(smem) + (threadIdx.x >> 3);
    const NodeRay nr = node_ray(ray);
    // row of the near planes per axis, and the lane's word in it
    const uint32_t word = (sub >> 1) * 4u;
    const uint32_t rowx = nr.rowx + word, rowy = nr.rowy + word, rowz = nr.rowz + word;
    TShear shear = make_shear(ray.d);
    shear.ox = shear_proj(ray.o, shear.bx);
    shear.oy = shear_proj(ray.o, shear.by);
    int sp = 0;
    uint32_t node = 0;   // the root
    while (__any_sync(ALL, active)) {
        __syncwarp();   // stack entries written in the last step are visible
        // ---- visit: the lane's child
        bool in = false;
        uint32_t vm = 0, tbase = 0, cbase = 0;
        if (active) {
            const uintptr_t np = reinterpret_cast<uintptr_t>(sv.nodes + node) ^ ((node & 7u) << 4);
            auto row = [&](uint32_t off) { return __ldg(reinterpret_cast<const float4*>(np ^ off)); };
            auto plane = [&](uint32_t off) {
                const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(np ^ off));
                return (sub & 1u) ? __half2float(__habs(__ushort_as_half((unsigned short)(w & 0xFFFFu)))) : __uint_as_float(w);
            };
            const float4 w0 = row(0x00u), w1 = row(0x10u);
            const float xn = plane(rowx), xf = plane(rowx ^ 0x70u), yn = plane(rowy), yf = plane(rowy ^ 0x50u),
                        zn = plane(rowz), zf = plane(rowz ^ 0x30u);
            if (COUNT) st.nodes += sub == 0;
            const uint32_t ew = __float_as_uint(w0.w);
            const float sx = __uint_as_float(ew & 0x7F800000u) * nr.idir.x;
            const float sy = __uint_as_float((ew << 8) & 0x7F800000u) * nr.idir.y;
            const float sz = __uint_as_float((ew << 16) & 0x7F800000u) * nr.idir.z;
            const float ax = fmaf(-256.0f, sx, fmaf(w0.x, nr.idir.x, nr.ood.x));
            const float ay = fmaf(-256.0f, sy, fmaf(w0.y, nr.idir.y, nr.ood.y));
            const float az = fmaf(-256.0f, sz, fmaf(w0.z, nr.idir.z, nr.ood.z));
            const float gap = fminf(fminf(fmaf(xf, sx, ax), fmaf(yf, sy, ay)), fminf(fmaf(zf, sz, az), ray.tmax)) -
                              fmaxf(fmaxf(fmaf(xn, sx, ax), fmaf(yn, sy, ay)), fmaxf(fmaf(zn, sz, az), ray.tmin));
            in = !(__float_as_uint(gap) >> 31);
            cbase = __float_as_uint(w1.x);
            tbase = __float_as_uint(w1.y);
            vm = __float_as_uint(w1.z);
        }
        const uint32_t hits = (__ballot_sync(ALL, in) >> oct0) & 0xFFu;
        const uint32_t tvalid = vm & 0x00FFFFFFu;
        uint32_t tmask = leaf_bits(hits) & tvalid;
        // ---- next internal node (a nearer hit does not change which)
        uint2 group = make_uint2(cbase, ((hits << 24) & vm) | (vm >> 24));
        bool more = active;
        if (active && group.y <= 0x00FFFFFFu) {
            more = sp != 0;
            if (more) group = stack[--sp * OCT_RAYS];
        }
        __syncwarp();   // the entry has been read by the ray's lanes before it may be overwritten
        if (more) {
            node = next_child(group, nr);
            if (group.y > 0x00FFFFFFu) {
                if (sp < CRT_STACK_TOTAL) {
                    if (sub == 0) stack[sp * OCT_RAYS] = group;
                    ++sp;
                } else {
                    if (sub == 0) atomicOr(err, (uint32_t)DEVERR_STACK_OVERFLOW);
                    more = false;
                }
            }
        }
        // ---- leaf triangles of the visited node, eight at a time: lane k takes the k-th
        while (__any_sync(ALL, tmask != 0u)) {
            uint32_t m = tmask;
            for (uint32_t k = 0; k < sub; ++k) m &= m - 1u;   // (0 stays 0)
            const uint32_t low = m & (0u - m);
            bool ok = false;
            float t = 0.f, wv = 0.f, ww = 0.f, dt = 1.f;
            uint32_t slot = 0;
            if (m) {
                slot = tbase + __popc(tvalid & (low - 1u));
                if (slot != ray.skip) {
                    const float4* tp = sv.tris + 3ull * slot;
                    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                    if (COUNT) st.tris++;
                    ok = tri_test(a, b, c, ray, shear, t, wv, ww, dt);
                }
            }
            const uint32_t any = (__ballot_sync(ALL, ok) >> oct0) & 0xFFu;
            if (ANY) {
                if (any) {
                    hit.slot = 0;
                    more = false;
                    tmask = 0;
                }
            } else if (__any_sync(ALL, ok)) {
                float best = ok ? t : __uint_as_float(0x7F800000u);   // (+inf may be a hit's distance)
                for (int o = 1; o < 8; o <<= 1) best = fminf(best, __shfl_xor_sync(ALL, best, o));
                const uint32_t win = (__ballot_sync(ALL, ok && t == best) >> oct0) & 0xFFu;
                const int from = (int)oct0 + (win ? 31 - __clz(win) : 0);
                const float u = __shfl_sync(ALL, wv, from), v = __shfl_sync(ALL, ww, from);
                const float d = __shfl_sync(ALL, dt, from);
                const uint32_t sl = __shfl_sync(ALL, slot, from);
                if (win) {
                    ray.tmax = not_neg0(best);
                    hit.u = u;
                    hit.v = v;
                    det = d;
                    hit.slot = sl;
                }
            }
            for (int k = 0; k < 8; ++k) tmask &= tmask - 1u;
        }
        active = more;
    }
    if (ANY) return hit;
    const float inv = 1.0f / det;
    hit.t = hit.slot != CRT_MISS ? ray.tmax : 0.0f;
    hit.u *= inv;
    hit.v *= inv;
    return hit;
}
