// Query kernels over one compressed 8-wide BVH (layout.h): unsigned distance,
// the two sign passes of signed distance (watertight / raystab), and
// closest-hit ray tracing.
//
// Reference kernels replaced: src/bvh.cu:631-740 and the traversals they
// call (src/bvh.cu:250-427): one thread per query, 128-thread blocks, a
// 32-entry local stack, children re-sorted per visit.
//
// Execution model here:
//  * point queries are visited in Morton-cell order (a counting sort of the
//    points into 2^(3b) cells of their bounding box), 32 neighbouring ones a
//    packet; the permutation only reorders work, every result is written to
//    the query's own index;
//  * a warp walks the tree once per packet with warp-uniform control flow
//    (k_udf, k_ray); persistent warps draw packets from a queue;
//  * queries and rays that do not fit packets (long searches, incoherent
//    rays, stab rays) are walked by a warp or a lane each.
#include <climits>
#include <cstdint>
#include <cooperative_groups.h>
#include <cub/block/block_radix_sort.cuh>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "launches.h"
#include "geom.cuh"
#include "kernels.h"
#include "scan.cuh"

namespace cubvh {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kQBlock = 128;  // threads per block of the query kernels

// ------------------------------------------------------------------ nodes
struct NodeView {
    float ox, oy, oz, sx, sy, sz;
    int child_base, tri_base;
    uint32_t meta0, meta1;
    uint32_t lx0, lx1, ly0, ly1, lz0, lz1, hx0, hx1, hy0, hy1, hz0, hz1;
};

__device__ __forceinline__ NodeView load_node(const CNode* __restrict__ nodes, int i) {
    const uint4* p = reinterpret_cast<const uint4*>(nodes + i);
    const uint4 w0 = __ldg(p), w1 = __ldg(p + 1), w2 = __ldg(p + 2), w3 = __ldg(p + 3), w4 = __ldg(p + 4);
    NodeView n;
    n.ox = __uint_as_float(w0.x); n.oy = __uint_as_float(w0.y); n.oz = __uint_as_float(w0.z);
    n.sx = exp2i((int)(int8_t)(w0.w & 0xFF));
    n.sy = exp2i((int)(int8_t)((w0.w >> 8) & 0xFF));
    n.sz = exp2i((int)(int8_t)((w0.w >> 16) & 0xFF));
    n.child_base = (int)w1.x; n.tri_base = (int)w1.y; n.meta0 = w1.z; n.meta1 = w1.w;
    n.lx0 = w2.x; n.lx1 = w2.y; n.ly0 = w2.z; n.ly1 = w2.w;
    n.lz0 = w3.x; n.lz1 = w3.y; n.hx0 = w3.z; n.hx1 = w3.w;
    n.hy0 = w4.x; n.hy1 = w4.y; n.hz0 = w4.z; n.hz1 = w4.w;
    return n;
}
template <class N>
__device__ __forceinline__ uint32_t meta_of(const N& n, int j) {
    return ((j < 4 ? n.meta0 : n.meta1) >> (8 * (j & 3))) & 0xFFu;
}
// Pairs of floats in one 64-bit register and the packed operations on them
// (two results per issued instruction), and the three-input maximum.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2unpack(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 f2add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ f2 f2max3(f2 a, f2 b, float c) {
    float a0, a1, b0, b1;
    f2unpack(a, a0, a1);
    f2unpack(b, b0, b1);
    return f2pack(max3(a0, b0, c), max3(a1, b1, c));
}

// byte k of w as a float: 0x4B0000qq is 2^23 + q, minus 2^23 is q exactly
__device__ __forceinline__ float qbyte(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + (unsigned)k)) - 8388608.0f;
}
// bytes k and k + 1 of w as floats
__device__ __forceinline__ f2 qpair(uint32_t w, int k) {
    const f2 q = f2pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + (unsigned)k)),
                        __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7541u + (unsigned)k)));
    return f2add(q, f2pack(-8388608.0f, -8388608.0f));
}
// origin + q * 2^e: exact product, one rounding (same as the host check)
__device__ __forceinline__ void child_box(const NodeView& n, int j, float3& lo, float3& hi) {
    const int b = j & 3;
    const bool h = j >= 4;
    lo.x = fmaf(qbyte(h ? n.lx1 : n.lx0, b), n.sx, n.ox);
    lo.y = fmaf(qbyte(h ? n.ly1 : n.ly0, b), n.sy, n.oy);
    lo.z = fmaf(qbyte(h ? n.lz1 : n.lz0, b), n.sz, n.oz);
    hi.x = fmaf(qbyte(h ? n.hx1 : n.hx0, b), n.sx, n.ox);
    hi.y = fmaf(qbyte(h ? n.hy1 : n.hy0, b), n.sy, n.oy);
    hi.z = fmaf(qbyte(h ? n.hz1 : n.hz0, b), n.sz, n.oz);
}
// >= 0: internal node index; < 0: leaf, -(slot * 4 + count - 1) - 1
template <class N>
__device__ __forceinline__ int child_ref(const N& n, uint32_t m) {
    if (m & 0x80u) return n.child_base + (int)(m & 7u);
    return -((((n.tri_base + (int)(m & 31u)) << 2) | (int)((m >> 5) & 3u)) + 1);
}

// Batcher odd-even merge sort network for 8 keys (19 comparators), ascending.
#define CUBVH_CS(i, j) { const uint32_t a_ = k[i], b_ = k[j]; k[i] = min(a_, b_); k[j] = max(a_, b_); }
__device__ __forceinline__ void sort8(uint32_t k[8]) {
    CUBVH_CS(0, 1) CUBVH_CS(2, 3) CUBVH_CS(4, 5) CUBVH_CS(6, 7)
    CUBVH_CS(0, 2) CUBVH_CS(1, 3) CUBVH_CS(4, 6) CUBVH_CS(5, 7)
    CUBVH_CS(1, 2) CUBVH_CS(5, 6)
    CUBVH_CS(0, 4) CUBVH_CS(1, 5) CUBVH_CS(2, 6) CUBVH_CS(3, 7)
    CUBVH_CS(2, 4) CUBVH_CS(3, 5)
    CUBVH_CS(1, 2) CUBVH_CS(3, 4) CUBVH_CS(5, 6)
}
#undef CUBVH_CS

__device__ __forceinline__ float box_d2(float3 p, float3 lo, float3 hi) {
    const float dx = fmaxf(fmaxf(lo.x - p.x, p.x - hi.x), 0.f);
    const float dy = fmaxf(fmaxf(lo.y - p.y, p.y - hi.y), 0.f);
    const float dz = fmaxf(fmaxf(lo.z - p.z, p.z - hi.z), 0.f);
    return dx * dx + dy * dy + dz * dz;
}
// Conservative slab interval of a ray with a zero direction component (inv =
// +-inf): computed bounds widened by 1e-6 relative (each bound carries at most
// three roundings).  A ray with d.x == 0 stays in the x slab of a box for every
// t if lo.x <= o.x <= hi.x and never otherwise; (lo.x - o.x) * inv.x is +-inf
// except when the origin lies on the plane (0 * inf = NaN), which then counts as
// inside the slab.  The other components may be all but zero, and then the
// double test cannot tell whether a ray from a plane leaves the box there:
// below 1e-12 of the largest component (kParallel), a slab that is not behind
// the ray has no exit.
constexpr float kParallel = 1e-12f;
__device__ __forceinline__ void box_ray(float3 o, float3 inv, float3 lo, float3 hi, float& tn, float& tf) {
    float t0x = (lo.x - o.x) * inv.x, t1x = (hi.x - o.x) * inv.x;
    float t0y = (lo.y - o.y) * inv.y, t1y = (hi.y - o.y) * inv.y;
    float t0z = (lo.z - o.z) * inv.z, t1z = (hi.z - o.z) * inv.z;
    if (t0x != t0x) t0x = -inv.x;
    if (t1x != t1x) t1x = inv.x;
    if (t0y != t0y) t0y = -inv.y;
    if (t1y != t1y) t1y = inv.y;
    if (t0z != t0z) t0z = -inv.z;
    if (t1z != t1z) t1z = inv.z;
    const float ix = fabsf(inv.x), iy = fabsf(inv.y), iz = fabsf(inv.z);
    const float along = fminf(fminf(ix, iy), iz) * (1.f / kParallel);
    float fx = fmaxf(t0x, t1x), fy = fmaxf(t0y, t1y), fz = fmaxf(t0z, t1z);
    if (ix >= along && fx >= 0.f) fx = CUDART_INF_F;
    if (iy >= along && fy >= 0.f) fy = CUDART_INF_F;
    if (iz >= along && fz >= 0.f) fz = CUDART_INF_F;
    tn = fmaxf(fmaxf(fminf(t0x, t1x), fminf(t0y, t1y)), fminf(t0z, t1z));
    tf = fminf(fminf(fx, fy), fz);
    tn -= 1e-6f * fabsf(tn);
    tf += 1e-6f * fabsf(tf);
}
// 1/d per axis; a ray with an infinite reciprocal (a zero or
// subnormal direction component) is tested with box_ray, the others as in
// affine_node.
__device__ __forceinline__ float3 ray_inv(float3 d) { return make_float3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z); }
__device__ __forceinline__ bool ray_degenerate(float3 inv) { return isinf(inv.x) || isinf(inv.y) || isinf(inv.z); }
// 1/d with the hardware approximation (at most 1 ulp off: the 1e-6 margins
// cover it) for unit directions; zero and subnormal components
// give +-inf, as ray_inv.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float3 ray_inv_approx(float3 d) {
    return make_float3(rcp_approx(d.x), rcp_approx(d.y), rcp_approx(d.z));
}

// Any-hit traversal step: push the children of node nd that the ray (o, inv)
// enters within [0, cull].
__device__ __forceinline__ void push_ray_children(const NodeView& nd, float3 o, float3 inv, float cull, int* st,
                                                  int& sp) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t m = meta_of(nd, j);
        float3 lo, hi;
        child_box(nd, j, lo, hi);
        float tn, tf;
        box_ray(o, inv, lo, hi, tn, tf);
        if (m != kEmpty && tn <= tf && tf >= 0.f && tn <= cull) st[sp++] = child_ref(nd, m);
    }
}

// The same step for a ray without zero direction components, with the
// node's affine decode folded into the ray: along axis a the plane of byte q
// is met at t = (origin_a + q * s_a - o_a) * inv_a, computed as
// fma(q, A_a, B_a) with A_a = s_a * inv_a and B_a = (origin_a - o_a) * inv_a.
// Against the decoded plane (itself origin + q * s rounded once) this is off
// by less than 6 * 2^-24 * S_a, S_a = |origin_a * inv_a| + 255 |A_a| + |B_a|
// (inv from the hardware reciprocal, within 1 ulp), so entries are computed
// with B_a - E_a and exits with B_a + E_a, E_a = 1e-6 * S_a (about 16 * 2^-24
// * S_a).  The ray's direction signs fix which of a child's two planes is
// the near one on each axis, so no per-child min / max is needed.
struct AffineNode { f2 ax, ay, az, nbx, fbx, nby, fby, nbz, fbz; uint32_t nx[2], fx[2], ny[2], fy[2], nz[2], fz[2]; };
__device__ __forceinline__ AffineNode affine_node(const NodeView& nd, float3 o, float3 inv) {
    const float ax = nd.sx * inv.x, ay = nd.sy * inv.y, az = nd.sz * inv.z;
    const float bx = (nd.ox - o.x) * inv.x, by = (nd.oy - o.y) * inv.y, bz = (nd.oz - o.z) * inv.z;
    const float ex = 1e-6f * (fabsf(nd.ox * inv.x) + 255.f * fabsf(ax) + fabsf(bx));
    const float ey = 1e-6f * (fabsf(nd.oy * inv.y) + 255.f * fabsf(ay) + fabsf(by));
    const float ez = 1e-6f * (fabsf(nd.oz * inv.z) + 255.f * fabsf(az) + fabsf(bz));
    const bool px = inv.x >= 0.f, py = inv.y >= 0.f, pz = inv.z >= 0.f;
    AffineNode a;
    a.ax = f2pack(ax, ax); a.ay = f2pack(ay, ay); a.az = f2pack(az, az);
    a.nbx = f2pack(bx - ex, bx - ex); a.fbx = f2pack(bx + ex, bx + ex);
    a.nby = f2pack(by - ey, by - ey); a.fby = f2pack(by + ey, by + ey);
    a.nbz = f2pack(bz - ez, bz - ez); a.fbz = f2pack(bz + ez, bz + ez);
    // near / far quantised words per axis (children 0-3, 4-7)
    a.nx[0] = px ? nd.lx0 : nd.hx0; a.nx[1] = px ? nd.lx1 : nd.hx1;
    a.fx[0] = px ? nd.hx0 : nd.lx0; a.fx[1] = px ? nd.hx1 : nd.lx1;
    a.ny[0] = py ? nd.ly0 : nd.hy0; a.ny[1] = py ? nd.ly1 : nd.hy1;
    a.fy[0] = py ? nd.hy0 : nd.ly0; a.fy[1] = py ? nd.hy1 : nd.ly1;
    a.nz[0] = pz ? nd.lz0 : nd.hz0; a.nz[1] = pz ? nd.lz1 : nd.hz1;
    a.fz[0] = pz ? nd.hz0 : nd.lz0; a.fz[1] = pz ? nd.hz1 : nd.lz1;
    return a;
}
// Entry and exit (at most cull) of the ray in children 2 c and 2 c + 1:
// entered where entry <= exit and 0 <= exit.  A coordinate that is no number
// bounds nothing: such a ray enters what its other axes meet, and hits nothing.
__device__ __forceinline__ void affine_pair(const AffineNode& a, int c, float cull, float tn[2], float tf[2]) {
    const int h = c >> 1, b = 2 * (c & 1);
    float x0, x1, y0, y1, z0, z1;
    f2unpack(f2fma(qpair(a.nx[h], b), a.ax, a.nbx), x0, x1);
    f2unpack(f2fma(qpair(a.ny[h], b), a.ay, a.nby), y0, y1);
    f2unpack(f2fma(qpair(a.nz[h], b), a.az, a.nbz), z0, z1);
    tn[0] = max3(x0, y0, z0);
    tn[1] = max3(x1, y1, z1);
    f2unpack(f2fma(qpair(a.fx[h], b), a.ax, a.fbx), x0, x1);
    f2unpack(f2fma(qpair(a.fy[h], b), a.ay, a.fby), y0, y1);
    f2unpack(f2fma(qpair(a.fz[h], b), a.az, a.fbz), z0, z1);
    tf[0] = fminf(min3(x0, y0, z0), cull);
    tf[1] = fminf(min3(x1, y1, z1), cull);
}
__device__ __forceinline__ void push_ray_children_affine(const NodeView& nd, float3 o, float3 inv, float cull,
                                                         int* st, int& sp) {
    const AffineNode a = affine_node(nd, o, inv);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float tn[2], tf[2];
        affine_pair(a, c, cull, tn, tf);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t m = meta_of(nd, 2 * c + i);
            if (m != kEmpty && tn[i] <= tf[i] && tf[i] >= 0.f) st[sp++] = child_ref(nd, m);
        }
    }
}

// Closest-hit step of one lane's own walk: entry distance (ordered bits of
// max(tn, 0), child index in the low 3 bits) of the ray into each child of
// nd that it enters within [0, cull], kFull for the others.  degen (a zero
// or subnormal direction component): box_ray on the decoded boxes;
// else the affine fold of push_ray_children_affine (same error margins).
__device__ __forceinline__ void lane_child_keys(const NodeView& nd, float3 o, float3 inv, bool degen, float cull,
                                                uint32_t k[8]) {
    if (degen) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float3 lo, hi;
            child_box(nd, j, lo, hi);
            float tn, tf;
            box_ray(o, inv, lo, hi, tn, tf);
            const float key = fmaxf(tn, 0.f);
            const bool need = meta_of(nd, j) != kEmpty && tn <= tf && tf >= 0.f && key <= cull;
            k[j] = need ? ((__float_as_uint(key) & ~7u) | (uint32_t)j) : kFull;
        }
        return;
    }
    const AffineNode a = affine_node(nd, o, inv);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float tn[2], tf[2];
        affine_pair(a, c, cull, tn, tf);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 2 * c + i;
            const bool need = meta_of(nd, j) != kEmpty && tn[i] <= tf[i] && tf[i] >= 0.f;
            k[j] = need ? ((__float_as_uint(fmaxf(tn[i], 0.f)) & ~7u) | (uint32_t)j) : kFull;
        }
    }
}
__device__ __forceinline__ float cull_of(double best) { return __double2float_ru(dM(best, 1.000001)); }
__device__ __forceinline__ void leaf_range(int ref, int& s0, int& s1) {
    const int code = -ref - 1;
    s0 = code >> 2; s1 = s0 + (code & 3) + 1;
}


// Dynamic packet queue: a warp takes `grab` consecutive 32-query packets per
// atomicAdd on a per-launch counter (zeroed before the launch), so warps that
// drew cheap packets keep taking more and no SM idles while work remains.
//
// Block budget (left != nullptr): the block's warps take at most *left grabs
// between them (a shared-memory count), then stop, and the block exits.  A
// launch of many such blocks (yield_shape) drains the same queue in short
// block lifetimes, so blocks of kernels on higher-priority streams get SMs
// between them instead of waiting for the whole launch.
struct PacketQueue {
    unsigned long long* ctr;
    int64_t npk, grab, next, end;
    int* left;
    __device__ __forceinline__ PacketQueue(unsigned long long* c, int64_t npk_, int64_t g, int* left_ = nullptr)
        : ctr(c), npk(npk_), grab(g), next(0), end(0), left(left_) {}
    __device__ __forceinline__ unsigned long long grab_start() {
        if (left && atomicSub(left, 1) <= 0) return (unsigned long long)npk;  // budget spent: done
        return atomicAdd(ctr, (unsigned long long)grab);
    }
    // index of the warp's next packet, or -1 when done
    __device__ __forceinline__ int64_t take() {
        if (next == end) {
            unsigned long long b = 0;
            if ((threadIdx.x & 31) == 0) b = grab_start();
            next = (int64_t)__shfl_sync(kFull, b, 0);
            end = next + grab;
        }
        const int64_t p = next++;
        return p < npk ? p : -1;
    }
    // the warp's next range of packets [b, e), false when done (warp-collective)
    __device__ __forceinline__ bool take_range(int64_t& b, int64_t& e) {
        unsigned long long v = 0;
        if ((threadIdx.x & 31) == 0) v = grab_start();
        b = (int64_t)__shfl_sync(kFull, v, 0);
        e = b + grab < npk ? b + grab : npk;
        return b < npk;
    }
};

// How k_udf's packets are handed out: tickets 0 .. nbig - 1 are `big`
// consecutive packets each, the later ones `grab`.  Warps that draw runs of
// neighbouring packets carry the seed from one to the next, and the short
// ones at the end even out what the packets cost.
struct RunShape {
    int64_t nbig, big, grab;
    // tickets that hand out npk packets
    __host__ __device__ int64_t tickets(int64_t npk) const {
        const int64_t rest = npk - nbig * big;
        return nbig + (rest > 0 ? (rest + grab - 1) / grab : 0);
    }
};
// The same queue over tickets (one atomicAdd each); block budget as above.
struct RunQueue {
    unsigned long long* ctr;
    int64_t npk, next, end;
    RunShape sh;
    int* left;
    __device__ __forceinline__ RunQueue(unsigned long long* c, int64_t npk_, RunShape s, int* left_)
        : ctr(c), npk(npk_), next(0), end(0), sh(s), left(left_) {}
    __device__ __forceinline__ int64_t take() {
        if (next == end) {
            unsigned long long v = ~0ull;
            if ((threadIdx.x & 31) == 0 && !(left && atomicSub(left, 1) <= 0)) v = atomicAdd(ctr, 1ull);
            v = __shfl_sync(kFull, v, 0);
            if (v == ~0ull) return -1;   // budget spent: done
            const int64_t t = (int64_t)v;
            next = t < sh.nbig ? t * sh.big : sh.nbig * sh.big + (t - sh.nbig) * sh.grab;
            end = next + (t < sh.nbig ? sh.big : sh.grab);
        }
        const int64_t p = next++;
        return p < npk ? p : -1;
    }
};

// What a launch works on: implicit 32-query packets over one BVH (root node
// 0), or a table of packets, each up to 32 consecutive positions of the
// query order on one mesh of an arena (root node, face-0 slot and first
// query index of that mesh).
struct Work {
    const PacketDesc* table;  // nullptr: implicit packets
    const MeshDesc* meshes;
    int64_t n;                // implicit: queries; table: packets
    int slot0;                // implicit: face-0 slot of the single BVH
    int64_t qbase = 0;        // implicit: index of query 0 within its call (raystab streams)
    __host__ __device__ __forceinline__ int64_t packets() const { return table ? n : (n + 31) >> 5; }
    // mesh of packet p (0: the single BVH)
    __device__ __forceinline__ int mesh_of(int64_t p) const { return table ? table[p].mesh : 0; }
    __device__ __forceinline__ void get(int64_t p, int64_t& start, int& count, int& root, int& s0,
                                        int64_t& qoff) const {
        if (table) {
            const PacketDesc d = table[p];
            const MeshDesc m = meshes[d.mesh];
            start = d.start; count = d.count; root = m.root; s0 = m.slot0; qoff = m.qoff;
        } else {
            start = p * 32; count = (int)min((int64_t)32, n - start); root = 0; s0 = slot0; qoff = -qbase;
        }
    }
};

__device__ __forceinline__ float3 load3(const float* __restrict__ a, int64_t i) {
    return make_float3(a[3 * i], a[3 * i + 1], a[3 * i + 2]);
}

// ------------------------------------------------------- unsigned distance
// ------------------------------------------------------- expanded records
// One thread per (node, child): the child's box as floats (layout.h, WNode).
__global__ void k_expand_nodes(int64_t n, const CNode* __restrict__ nodes, const CTri* __restrict__ tris,
                               WNode* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 8 * n) return;
    const int i = (int)(t >> 3), j = (int)(t & 7);
    const NodeView nd = load_node(nodes, i);
    const uint32_t m = meta_of(nd, j);
    float3 lo = make_float3(CUDART_INF_F, CUDART_INF_F, CUDART_INF_F);
    float3 hi = make_float3(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
    int ref = 0;
    if (m != kEmpty) {
        ref = child_ref(nd, m);
        if (ref >= 0) {
            float3 clo, chi;
            child_box(nd, j, clo, chi);
            const NodeView c = load_node(nodes, ref);
            for (int k = 0; k < 8; ++k) {
                if (meta_of(c, k) == kEmpty) continue;
                float3 l, h;
                child_box(c, k, l, h);
                lo = make_float3(fminf(lo.x, l.x), fminf(lo.y, l.y), fminf(lo.z, l.z));
                hi = make_float3(fmaxf(hi.x, h.x), fmaxf(hi.y, h.y), fmaxf(hi.z, h.z));
            }
            lo = make_float3(fmaxf(lo.x, clo.x), fmaxf(lo.y, clo.y), fmaxf(lo.z, clo.z));
            hi = make_float3(fminf(hi.x, chi.x), fminf(hi.y, chi.y), fminf(hi.z, chi.z));
        } else {
            const int code = -ref - 1;
            const int s0 = code >> 2, s1 = s0 + (code & 3) + 1;
            for (int s = s0; s < s1; ++s) {
                const TriV v = load_tri(tris, s);
                lo.x = fminf(lo.x, fminf(v.a.x, fminf(v.b.x, v.c.x)));
                lo.y = fminf(lo.y, fminf(v.a.y, fminf(v.b.y, v.c.y)));
                lo.z = fminf(lo.z, fminf(v.a.z, fminf(v.b.z, v.c.z)));
                hi.x = fmaxf(hi.x, fmaxf(v.a.x, fmaxf(v.b.x, v.c.x)));
                hi.y = fmaxf(hi.y, fmaxf(v.a.y, fmaxf(v.b.y, v.c.y)));
                hi.z = fmaxf(hi.z, fmaxf(v.a.z, fmaxf(v.b.z, v.c.z)));
            }
        }
    }
    float4* o = reinterpret_cast<float4*>(out + i);
    o[j] = make_float4(lo.x, lo.y, lo.z, __int_as_float(ref));
    o[8 + j] = make_float4(hi.x, hi.y, hi.z, 0.f);
}

// One thread per triangle: its frame (layout.h, WTri), in double.  A corner
// closer to the longest edge than 1e-9 of its length counts as on it.
__global__ void k_expand_tris(int64_t n, const CTri* __restrict__ tris, WTri* __restrict__ out) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const TriV t = load_tri(tris, (int)s);
    float3 A = t.a, B = t.b, C = t.c;
    const d3 eab = dsub(to_d3(B), to_d3(A)), ebc = dsub(to_d3(C), to_d3(B)), eca = dsub(to_d3(A), to_d3(C));
    const double lab = ddot(eab, eab), lbc = ddot(ebc, ebc), lca = ddot(eca, eca);
    d3 e = eab;
    double l2 = lab;
    if (lbc > lab && lbc >= lca) { A = t.b; B = t.c; C = t.a; e = ebc; l2 = lbc; }
    else if (lca > lab) { A = t.c; B = t.a; C = t.b; e = eca; l2 = lca; }
    const double L = sqrt(l2);
    const d3 ex = L > 0.0 ? dscale(e, 1.0 / L) : d3{1.0, 0.0, 0.0};
    const d3 w = dsub(to_d3(C), to_d3(A));
    const double cx = ddot(w, ex);
    d3 r = dsub(w, dscale(ex, cx));
    double cy = sqrt(ddot(r, r));
    d3 ey;
    if (cy > 1e-9 * L) {
        ey = dscale(r, 1.0 / cy);
        ey = dsub(ey, dscale(ex, ddot(ey, ex)));
    } else {
        cy = 0.0;
        const double ax = fabs(ex.x), ay = fabs(ex.y), az = fabs(ex.z);
        const d3 u = ax <= ay && ax <= az ? d3{1.0, 0.0, 0.0} : (ay <= az ? d3{0.0, 1.0, 0.0} : d3{0.0, 0.0, 1.0});
        ey = dcross(u, ex);
    }
    ey = dscale(ey, 1.0 / sqrt(ddot(ey, ey)));
    const double ac = sqrt(cx * cx + cy * cy), bx = cx - L, bc = sqrt(bx * bx + cy * cy);
    float4* o = reinterpret_cast<float4*>(out + s);
    // a triangle without a usable plane (K >= 1e9, layout.h: the sine of an angle below 1e-8, zero area
    // among them) is left undecided by an infinite length: the double evaluation's own rounding
    // could pass the filter's bound there, and gives no number at all for a repeated vertex
    o[0] = make_float4(A.x, A.y, A.z, t.k >= 1e9f ? CUDART_INF_F : (float)L);
    o[1] = make_float4((float)ex.x, (float)ex.y, (float)ex.z, (float)ac);
    o[2] = make_float4((float)ey.x, (float)ey.y, (float)ey.z, (float)bc);
    o[3] = make_float4(ac > 0.0 ? (float)(cx / ac) : 1.f, ac > 0.0 ? (float)(cy / ac) : 0.f,
                       bc > 0.0 ? (float)(bx / bc) : 1.f, bc > 0.0 ? (float)(cy / bc) : 0.f);
}

cudaError_t launch_expand(int64_t n_nodes, int64_t n_tris, const CNode* nodes, const CTri* tris, WNode* wnodes,
                          WTri* wtris, cudaStream_t stream) {
    if (n_nodes > 0) { k_expand_nodes<<<(unsigned)((8 * n_nodes + 255) / 256), 256, 0, stream>>>(n_nodes, nodes, tris, wnodes); count_launch(); }
    if (n_tris > 0) { k_expand_tris<<<(unsigned)((n_tris + 127) / 128), 128, 0, stream>>>(n_tris, tris, wtris); count_launch(); }
    return cudaGetLastError();
}

__device__ __forceinline__ TriW make_triw(float4 w0, float4 w1, float4 w2, float4 w3) {
    TriW t;
    t.a = make_float3(w0.x, w0.y, w0.z); t.len = w0.w;
    t.ex = make_float3(w1.x, w1.y, w1.z); t.lac = w1.w;
    t.ey = make_float3(w2.x, w2.y, w2.z); t.lbc = w2.w;
    t.vx = w3.x; t.vy = w3.y; t.ux = w3.z; t.uy = w3.w;
    return t;
}
constexpr int kCand = 8;            // candidate list of a query
constexpr int kUdfBlocks = 7;       // blocks of k_udf per SM

// Lower bound of the squared distance of p to the triangle in slot s.
__device__ __forceinline__ float tri_lower_bound(const WTri* __restrict__ wtris, int s, float3 p) {
    const float4* tw = reinterpret_cast<const float4*>(wtris + s);
    float err;
    const float d2 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
    return d2 - err;
}

// Exact nearest triangles of the points of a packet's lanes `on`, given upper
// bounds U of their squared distances, as the only entries of their lists (32
// entries apart): the warp walks the union of their paths once more, and each
// lane evaluates in double every triangle whose lower bound is within its U.
// The bounds that k_udf's walk ends with are all but exact, so this meets
// little more than the triangles that tie.  Returns the list's length.
__device__ __noinline__ int walk_ties(const WNode* __restrict__ wnodes, const WTri* __restrict__ wtris,
                                      const CTri* __restrict__ tris, uint2* stk, uint2* cand, int root, float3 p, float U,
                                      bool on) {
    double best = 1e6;
    int slot = -1, id = 0;
    int sp = 0, cur = root;
    while (true) {
        if (cur >= 0) {
            const float4* nb = reinterpret_cast<const float4*>(wnodes + cur);
            const float cull = on ? U * 1.000002f : -1.f;
            __syncwarp();   // the popped entry has been read
            for (int j = 0; j < 8; ++j) {
                const float4 lo = __ldg(nb + j), hi = __ldg(nb + 8 + j);
                if (__any_sync(kFull, box_d2(p, make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z)) <= cull)) {
                    if ((threadIdx.x & 31) == 0) stk[sp].x = (uint32_t)__float_as_int(lo.w);
                    ++sp;
                }
            }
            __syncwarp();
        } else {
            int s0, s1;
            leaf_range(cur, s0, s1);
            for (int s = s0; s < s1; ++s) {
                const float4* tw = reinterpret_cast<const float4*>(wtris + s);
                float err;
                const float d2 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
                if (!on || d2 - err > U) continue;   // no number: undecided
                const TriV t = load_tri(tris, s);
                const double e = dist2_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c));
                if (e < best || (e == best && (slot < 0 || t.id < id))) { best = e; slot = s; id = t.id; }
            }
            if (slot >= 0) U = fminf(U, __double2float_ru(best));
            __syncwarp();
        }
        if (sp == 0) break;
        cur = (int)stk[--sp].x;
    }
    if (slot < 0) return 0;
    cand[0] = make_uint2((uint32_t)slot, __float_as_uint(0.f));
    return 1;
}

// Exact nearest triangle of 32 Morton-adjacent points per warp (a packet):
// the warp walks the union of the lanes' search paths with warp-uniform
// control flow.  At an inner node, lane 8 g + j tests child j against the
// eight points of group g (8 consecutive points of the packet, kept in the
// registers of all the group's lanes): a child is needed when its box is
// within the bound of some point.  So the lanes read different boxes (two
// coalesced 16-byte loads a node) and reduce over points in registers, two
// points an instruction: about 92 instructions a node.  With a lane per
// point, every lane reads all eight boxes (64 cycles of the SM's load path a
// node, which became the bound) and each child needs a warp minimum: 180
// instructions.  Bounding the groups by boxes instead of testing their
// points keeps ten times the leaves.  The warp's stack and the candidate
// lists are in shared memory: 72 registers, 28 warps per SM (16 warps: 10 %
// slower).  The lane's winner of the warp's previous packet, next to this
// one in Morton order, gives the first bound.
// Children are pushed farthest first (by the smallest distance of any point).
// Leaves run the FP32 triangle test in every lane; each lane
// keeps U, an upper bound of its squared distance (FP32 estimate + its error
// bound), and a short list of triangles whose lower bound is within U.  At
// the end every lane evaluates its surviving candidates in double: the
// minimum (ties -> lowest face index) is the exact nearest triangle.
//
// A point that is not finite, or farther than MAX_DIST from the root's box,
// finds nothing and takes no part in the walk.
//
// Bound by instruction issue and the latency of node and triangle loads; at 72
// registers each variant spills 240 bytes of stores and 210 of loads.  Measured against the walk with a
// lane per point and the records of layout.h's first half, whole calls: 1M
// points on 5,120 faces 1.98 -> 0.99 ms, 384^3 grid on 177k faces 107.5 -> 48.0
// ms, 8.4M watertight points on 82k faces 9.70 -> 5.52 ms.
//
// Heavy queries, served afterwards with a warp each (k_udf_heavy, from the
// bound found so far): a point whose candidate list overflows (many
// triangles at almost the same distance) in a packet with fewer than
// kTiesHere of them, and the points of a packet that
// is still walking after kHandOff visits when the queue is empty: deep
// inside a closed mesh or near its medial axis points are about equally far
// from very many triangles, and such a packet would hold the launch's end
// alone.  Only while few packets do so (kLateMost, counted from kLate visits
// on): a warp a query is for idle SMs, and when most of a launch is such
// packets it is many times the work (100,003 points at one place in 1.3M
// faces 1,550 -> 567 us, within 0.1 of it 888 -> 678; a limit of 640 gives 569
// and 526, but uniform points 820, 681 before and 672 at 1,500).  After
// kHandOffAny visits packets are handed off in any case: the 384^3 grid has
// unions of thousands of visits, 57 ms without that line, 51 at 1,024, 50.0 at 512.
// When the heavy list is full both finish here instead, as do the
// points of a packet most of which tie (faces that are there several times):
// walked together once more they cost a fraction of a warp each (300k points
// on 12 copies of 5,120 faces 36 against 5.1 ms, 1M at the middle of 3 copies
// of 82k faces 7.7 against 5.5).  The grid of 384^3 points has packets of both
// kinds and pays 2 % (48.9 against 50.0 ms); lines of 4 to 28 points measure
// the same, so the line is a quarter of the packet.
constexpr int kLate = 128, kHandOff = 192, kHandOffAny = 512;
constexpr int kLateMost = 1500;
constexpr int kTiesHere = 8;
template <bool UVW, bool SLOT>
__global__ void __launch_bounds__(kQBlock, kUdfBlocks) k_udf(Work w, const uint32_t* __restrict__ order,
                                                 const float* __restrict__ pts, float* __restrict__ dist,
                                                 int64_t* __restrict__ face_id, float* __restrict__ uvw,
                                                 int32_t* __restrict__ slot_out, const DeviceTree tree,
                                                 unsigned long long* __restrict__ ctr, RunShape shape,
                                                 uint4* __restrict__ heavy, unsigned long long* __restrict__ n_heavy,
                                                 int64_t heavy_cap, unsigned long long* __restrict__ late,
                                                 int block_grabs) {
    const CTri* __restrict__ tris = tree.tris;
    const int lane = threadIdx.x & 31;
    __shared__ uint2 s_cand[kQBlock / 32][kCand][32];
    __shared__ uint2 s_stack[kQBlock / 32][kStack];
    __shared__ int s_left;
    uint2* cand = &s_cand[threadIdx.x >> 5][0][lane];   // the lane's candidates, 32 entries apart: slot, lower bound
    uint2* stk = s_stack[threadIdx.x >> 5];
    if (block_grabs > 0) {  // uniform: the launch's block budget
        if (threadIdx.x == 0) s_left = block_grabs;
        __syncthreads();
    }
    RunQueue pq(ctr, w.packets(), shape, block_grabs > 0 ? &s_left : nullptr);
    const unsigned long long tickets = (unsigned long long)shape.tickets(w.packets());
    int seed = -1, seed_root = -1;   // the lane's winning slot in the warp's previous packet, and its tree
    for (int64_t pk = pq.take(); pk >= 0; pk = pq.take()) {
        int64_t start, qoff;
        int cnt, root, slot_face0;
        w.get(pk, start, cnt, root, slot_face0, qoff);
        const int64_t qi = start + lane;
        const bool act = lane < cnt;
        const int64_t idx = act ? (order ? (int64_t)order[qi] : qi) : 0;
        const float3 p = act ? load3(pts, idx) : make_float3(0.f, 0.f, 0.f);
        bool near_root;              // the point can be within MAX_DIST of the mesh
        {
            const CNode* rn = tree.nodes + root;
            const float3 lo = make_float3(rn->ox, rn->oy, rn->oz);
            const float3 hi = make_float3(fmaf(255.f, exp2i(rn->ex), lo.x), fmaf(255.f, exp2i(rn->ey), lo.y),
                                          fmaf(255.f, exp2i(rn->ez), lo.z));
            near_root = act && isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && box_d2(p, lo, hi) <= 1e6f * 1.000002f;
        }
        // U: upper bound of the lane's nearest squared distance (MAX_DIST^2)
        float U = near_root ? 1e6f : -1.f;
        if (root == seed_root && near_root && seed >= 0) {
            const float4* tw = reinterpret_cast<const float4*>(tree.wtris + seed);
            float err;
            const float e32 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
            U = fminf(U, e32 + err);
        }
        int nc = 0;
        // the group's points (infinitely far where there is none) and their bounds, in pairs
        f2 gx[4], gy[4], gz[4];
        float gc[8];
        uint32_t cullmax;
        {
            const float3 q = near_root ? p : make_float3(CUDART_INF_F, CUDART_INF_F, CUDART_INF_F);
            const int g0 = lane & 24;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                gx[i] = f2pack(__shfl_sync(kFull, q.x, g0 + 2 * i), __shfl_sync(kFull, q.x, g0 + 2 * i + 1));
                gy[i] = f2pack(__shfl_sync(kFull, q.y, g0 + 2 * i), __shfl_sync(kFull, q.y, g0 + 2 * i + 1));
                gz[i] = f2pack(__shfl_sync(kFull, q.z, g0 + 2 * i), __shfl_sync(kFull, q.z, g0 + 2 * i + 1));
            }
        }
        auto share_bounds = [&]() {
            const float cull = near_root ? U * 1.000002f : -1.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) gc[i] = __shfl_sync(kFull, cull, (lane & 24) + i);
            cullmax = __reduce_max_sync(kFull, __float_as_uint(fmaxf(cull, 0.f)));
        };
        share_bounds();
        const f2 p2[3] = {f2pack(p.x, p.x), f2pack(p.y, p.y), f2pack(p.z, p.z)};
        const f2 neg = f2pack(-1.f, -1.f);
        int sp = 0;
        int cur = root;
        bool live = __any_sync(kFull, near_root);
        int work = 0;
        bool handed_off = false, counted = false;
        while (live) {
            if ((++work & 63) == 0 && work >= kLate) {   // warp-uniform
                unsigned long long taken = 0, others = 0;
                if (lane == 0) {
                    taken = *reinterpret_cast<volatile unsigned long long*>(ctr);
                    if (taken >= tickets) others = counted ? *reinterpret_cast<volatile unsigned long long*>(late) : atomicAdd(late, 1ull);
                }
                taken = __shfl_sync(kFull, taken, 0);
                const bool first = !counted;
                counted = taken >= tickets;
                if (counted && !first && (work >= kHandOffAny || __shfl_sync(kFull, (int)others, 0) <= kLateMost)) {
                    unsigned long long b = 0;
                    if (lane == 0) b = atomicAdd(n_heavy, (unsigned long long)cnt);
                    b = __shfl_sync(kFull, b, 0);
                    const uint32_t mesh = w.table ? (uint32_t)w.table[pk].mesh : 0u;
                    // a list without room for all takes what fits; those queries are served twice, with the same result
                    if (act && (int64_t)b + lane < heavy_cap) heavy[b + lane] = make_uint4((uint32_t)idx, mesh, __float_as_uint(U), 0u);
                    if ((int64_t)b + cnt <= heavy_cap) { handed_off = true; break; }
                }
            }
            if (cur >= 0) {
                const float4* nb = reinterpret_cast<const float4*>(tree.wnodes + cur);
                const int j = lane & 7;
                const float4 lo = __ldg(nb + j), hi = __ldg(nb + 8 + j);
                const f2 lx = f2pack(lo.x, lo.x), ly = f2pack(lo.y, lo.y), lz = f2pack(lo.z, lo.z);
                const f2 hx = f2pack(-hi.x, -hi.x), hy = f2pack(-hi.y, -hi.y), hz = f2pack(-hi.z, -hi.z);
                bool need = false;
                float dmin = CUDART_INF_F;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f2 dx = f2max3(f2fma(gx[i], neg, lx), f2add(gx[i], hx), 0.f);
                    const f2 dy = f2max3(f2fma(gy[i], neg, ly), f2add(gy[i], hy), 0.f);
                    const f2 dz = f2max3(f2fma(gz[i], neg, lz), f2add(gz[i], hz), 0.f);
                    float da, db;
                    f2unpack(f2fma(dz, dz, f2fma(dy, dy, f2mul(dx, dx))), da, db);
                    need |= da <= gc[2 * i];
                    need |= db <= gc[2 * i + 1];
                    dmin = min3(dmin, da, db);
                }
                unsigned m = __ballot_sync(kFull, need);
                m = (m | (m >> 16));
                m = (m | (m >> 8)) & 0xFFu;          // needed children
                uint32_t key = __float_as_uint(dmin);
                key = min(key, __shfl_xor_sync(kFull, key, 8));
                key = min(key, __shfl_xor_sync(kFull, key, 16));
                key = (m >> j) & 1u ? ((key & ~7u) | (uint32_t)j) : kFull;
                // its place on the stack: the number of needed children farther than it, two of
                // the eight compared by each of the four lanes with this child
                const uint32_t ka = __shfl_sync(kFull, key, 2 * (lane >> 3)), kb = __shfl_sync(kFull, key, 2 * (lane >> 3) + 1);
                int pos = (ka > key && ka != kFull ? 1 : 0) + (kb > key && kb != kFull ? 1 : 0);
                pos += __shfl_xor_sync(kFull, pos, 8);
                pos += __shfl_xor_sync(kFull, pos, 16);
                const int kept = __popc(m);
                __syncwarp();   // the popped entry has been read
                if (lane < 8 && key != kFull) stk[sp + pos] = make_uint2((uint32_t)__float_as_int(lo.w), key & ~7u);
                sp += kept;
                __syncwarp();
            } else {
                int s0, s1;
                leaf_range(cur, s0, s1);
                const float U0 = U;
                const float4* tw = reinterpret_cast<const float4*>(tree.wtris + s0);
                for (int s = s0; s < s1; ++s, tw += 4) {
                    float err;
                    const float e32 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
                    const float lb = e32 - err;
                    const bool c = near_root && !(lb > U);   // within the bound, or undecided (no number)
                    if (c) {
                        U = fminf(U, e32 + err);
                        if (nc == kCand) {   // keep only live candidates
                            int m = 0;
                            for (int k = 0; k < kCand; ++k)
                                if (!(__uint_as_float(cand[32 * k].y) > U)) { cand[32 * m] = cand[32 * k]; ++m; }
                            nc = m < kCand ? m : kCand + 1;
                        }
                        if (nc < kCand) {
                            cand[32 * nc] = make_uint2((uint32_t)s, __float_as_uint(lb));
                            ++nc;
                        }   // else the list has overflowed (nc = kCand + 1)
                    }
                }
                if (__any_sync(kFull, U < U0)) share_bounds();
            }
            // the next entry that some point still needs
            live = false;
            while (sp > 0) {
                const uint2 e = stk[--sp];
                if (e.y <= cullmax) { cur = (int)e.x; live = true; break; }
            }
        }
        if (handed_off) continue;
        if (counted && lane == 0) atomicAdd(late, ~0ull);
        bool mine = act;
        const bool many = __popc(__ballot_sync(kFull, nc > kCand)) >= kTiesHere;
        bool again = false;
        if (nc > kCand) {
            const unsigned long long b = many ? (unsigned long long)heavy_cap : atomicAdd(n_heavy, 1ull);
            if ((int64_t)b < heavy_cap) {
                heavy[b] = make_uint4((uint32_t)idx, w.table ? (uint32_t)w.table[pk].mesh : 0u, __float_as_uint(U), 0u);
                mine = false;
            } else {
                again = true;
            }
            nc = 0;
        }
        if (__any_sync(kFull, again)) {
            const int left = walk_ties(tree.wnodes, tree.wtris, tris, stk, cand, root, p, U, again);
            if (again) nc = left;
        }
        double bx = 1e6;
        int sx = -1, ix = 0;
        // the k-th live candidates of all lanes together
        for (int i = 0;; ++i) {
            while (i < nc && __uint_as_float(cand[32 * i].y) > U) ++i;
            if (!__any_sync(kFull, i < nc)) break;
            if (i < nc) {
                const int s = (int)cand[32 * i].x;
                const TriV t = load_tri(tris, s);
                const double e = dist2_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c));
                if (e < bx || (e == bx && (sx < 0 || t.id < ix))) { bx = e; sx = s; ix = t.id; }
            }
        }
        seed = sx;
        seed_root = root;
        if (!mine) continue;
        double d64;
        if (sx < 0) {  // nothing within MAX_DIST: distance 0 on face 0
            sx = slot_face0; d64 = 0.0;
            ix = load_tri(tris, sx).id;
        } else {
            d64 = __dsqrt_rn(bx);
        }
        dist[idx] = __double2float_rn(d64);
        face_id[idx] = (int64_t)ix;
        if (SLOT) slot_out[idx] = sx;
        if (UVW) {
            const TriV t = load_tri(tris, sx);
            double bary[3]; d3 cp;
            closest_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c), bary, &cp);
            uvw[3 * idx] = __double2float_rn(bary[0]);
            uvw[3 * idx + 1] = __double2float_rn(bary[1]);
            uvw[3 * idx + 2] = __double2float_rn(bary[2]);
        }
    }
}


// ---------------------------------------------------------- heavy queries
// One warp per query handed off by k_udf.  Each step pops up to four live
// nodes from a stack in shared memory (lane = child j of popped node i,
// 8 * i + j), pushes the internal children within the bound and collects the
// triangles of the leaf children, which are tested when 32 of them are there
// (one per lane) or the stack is empty: a step brings 4 to 11 on average, and
// issue slots bound this kernel, so testing each step's own cost more than
// the later bound does (1M points on 5,120 faces 0.963 -> 0.923 ms a call,
// an arena of 48 meshes 3.58 -> 3.53, 1,000 points 57 -> 53 us).  U (an upper
// bound of the squared distance) and the candidate list are the warp's, and
// candidates are settled in double exactly as in k_udf, so the result is the
// same exact nearest triangle (lowest face index on ties).
constexpr int kHStack = 512;
constexpr int kHCand = 64;
// Each step pushes at most 32 children one level below the deepest node it
// popped, so the stack holds at most one such batch per tree level.
static_assert(kHStack >= 32 * (kMaxDepth + 1), "heavy-query stack too small for the tree depth");
struct HeavyWarp {
    int ref[kHStack];
    uint32_t key[kHStack];
    int pop[4];
    int tslot[31 + 4 * 32];   // what was left, and a step's leaves
    int cs[kHCand];
    float cl[kHCand];
};

// Exact minimum (ties -> lowest face index) over the candidates i < nc whose
// lower bound is <= lim, merged into (bx, sx, ix); warp-parallel, the result
// is the same in every lane.
__device__ void heavy_settle(const HeavyWarp& S, int nc, float lim, const CTri* __restrict__ tris, float3 p,
                             double& bx, int& sx, int& ix) {
    const int lane = threadIdx.x & 31;
    double e = CUDART_INF;
    int s = -1, id = INT_MAX;
    for (int i = lane; i < nc; i += 32) {
        if (S.cl[i] > lim) continue;
        const int sl = S.cs[i];
        const TriV t = load_tri(tris, sl);
        const double d = dist2_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c));
        if (d < e || (d == e && t.id < id)) { e = d; s = sl; id = t.id; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double e2 = __shfl_xor_sync(kFull, e, o);
        const int s2 = __shfl_xor_sync(kFull, s, o), id2 = __shfl_xor_sync(kFull, id, o);
        if (e2 < e || (e2 == e && id2 < id)) { e = e2; s = s2; id = id2; }
    }
    if (s >= 0 && (e < bx || (e == bx && (sx < 0 || id < ix)))) { bx = e; sx = s; ix = id; }
}

// The walk of one query by the whole warp: the exact nearest triangle of p
// under `root` into (bx, sx, ix), the same in every lane.  U: a bound of its
// squared distance (negative: nothing can be found).
__device__ void heavy_walk(HeavyWarp& S, const DeviceTree& tree, int root, float3 p, float U, double& bx, int& sx,
                           int& ix) {
    const CTri* __restrict__ tris = tree.tris;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int nc = 0, nt = 0, sp = U >= 0.f ? 1 : 0;
    U = fminf(1e6f, fmaxf(U, 0.f));   // MAX_DIST^2
    bx = 1e6;
    sx = -1;
    ix = 0;
    __syncwarp();  // the previous query is done with S
    if (lane == 0) { S.ref[0] = root; S.key[0] = 0u; }
    __syncwarp();
    while (sp > 0) {
        const float cull = U * 1.000002f;
        // pop: of the top 32 entries, the first four (from the top) whose
        // key is within the bound; the culled ones above them go too
        const int pos = sp - 1 - lane;
        const bool alive = pos >= 0 && S.key[pos] <= __float_as_uint(cull);
        const unsigned m = __ballot_sync(kFull, alive);
        int nn = __popc(m), used = sp < 32 ? sp : 32;
        if (nn >= 4) {  // up to and including the fourth live entry
            unsigned m4 = m;
            m4 &= m4 - 1u;
            m4 &= m4 - 1u;
            m4 &= m4 - 1u;
            used = __ffs(m4);
            nn = 4;
        }
        if (alive && __popc(m & lt) < 4) S.pop[__popc(m & lt)] = S.ref[pos];
        sp -= used;
        __syncwarp();
        // children of the popped nodes
        const int ni = lane >> 3, j = lane & 7;
        bool take = false, leaf = false;
        int cref = 0;
        uint32_t key = 0u;
        if (ni < nn) {
            const float4* nb = reinterpret_cast<const float4*>(tree.wnodes + S.pop[ni]);
            const float4 lo = __ldg(nb + j), hi = __ldg(nb + 8 + j);
            const float d2 = box_d2(p, make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z));
            if (d2 <= cull) {   // an unused child's box is infinitely far
                take = true;
                key = __float_as_uint(d2);
                cref = __float_as_int(lo.w);
                leaf = cref < 0;
            }
        }
        const unsigned mi = __ballot_sync(kFull, take && !leaf);
        if (take && !leaf) {
            const int q = sp + __popc(mi & lt);
            S.ref[q] = cref;
            S.key[q] = key;
        }
        sp += __popc(mi);
        // the leaf children's triangles
        const unsigned ml = __ballot_sync(kFull, take && leaf);
        if (ml) {
            int c = 0, a = 0;
            if (take && leaf) {
                int b;
                leaf_range(cref, a, b);
                c = b - a;                       // 1 to 4
            }
            const unsigned m0 = __ballot_sync(kFull, c > 0 && ((c - 1) & 1)), m1 = __ballot_sync(kFull, c > 0 && ((c - 1) & 2));
            const int at = nt + __popc(ml & lt) + __popc(m0 & lt) + 2 * __popc(m1 & lt);
            for (int i = 0; i < c; ++i) S.tslot[at + i] = a + i;
            nt += __popc(ml) + __popc(m0) + 2 * __popc(m1);
        }
        __syncwarp();  // the stack's new entries and the leaves' triangles
        int base = 0;
        for (; base + 32 <= nt || (sp == 0 && base < nt); base += 32) {
            const int t = base + lane;
            float e32 = 0.f, err = 0.f;
            int slot = -1;
            if (t < nt) {
                slot = S.tslot[t];
                const float4* tw = reinterpret_cast<const float4*>(tree.wtris + slot);
                e32 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
            }
            const float ub = t < nt ? e32 + err : CUDART_INF_F;
            U = fminf(U, __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(ub))));
            const float lb = e32 - err;
            const bool cand = t < nt && !(lb > U);
            const unsigned mc = __ballot_sync(kFull, cand);
            if (nc + __popc(mc) > kHCand) {  // warp-uniform: drop dead candidates, else settle them
                int keep = 0;
                for (int i0 = 0; i0 < nc; i0 += 32) {
                    const int i = i0 + lane;
                    const bool kp = i < nc && !(S.cl[i] > U);
                    const int cs_i = kp ? S.cs[i] : 0;
                    const float cl_i = kp ? S.cl[i] : 0.f;
                    const unsigned mk = __ballot_sync(kFull, kp);
                    __syncwarp();  // every lane has read its entry
                    if (kp) {
                        S.cs[keep + __popc(mk & lt)] = cs_i;
                        S.cl[keep + __popc(mk & lt)] = cl_i;
                    }
                    keep += __popc(mk);
                    __syncwarp();
                }
                nc = keep;
                if (nc + __popc(mc) > kHCand) {
                    heavy_settle(S, nc, CUDART_INF_F, tris, p, bx, sx, ix);
                    U = fminf(U, __double2float_ru(bx));
                    nc = 0;
                    __syncwarp();
                }
            }
            if (cand) {
                S.cs[nc + __popc(mc & lt)] = slot;
                S.cl[nc + __popc(mc & lt)] = lb;
            }
            nc += __popc(mc);
            __syncwarp();
        }
        if (base) {   // the rest to the front
            nt = max(nt - base, 0);
            const int left = lane < nt ? S.tslot[base + lane] : 0;
            __syncwarp();
            if (lane < nt) S.tslot[lane] = left;
            __syncwarp();
        }
    }
    heavy_settle(S, nc, U, tris, p, bx, sx, ix);
}

// Writes a query's result from its exact nearest triangle (sx < 0: none).
template <bool UVW, bool SLOT>
__device__ __forceinline__ void write_nearest(const CTri* __restrict__ tris, int64_t idx, float3 p, double bx, int sx,
                                              int ix, int slot_face0, float* __restrict__ dist,
                                              int64_t* __restrict__ face_id, float* __restrict__ uvw,
                                              int32_t* __restrict__ slot_out) {
    double d64;
    if (sx < 0) {  // nothing within MAX_DIST: distance 0 on face 0
        sx = slot_face0;
        d64 = 0.0;
        ix = load_tri(tris, sx).id;
    } else {
        d64 = __dsqrt_rn(bx);
    }
    dist[idx] = __double2float_rn(d64);
    face_id[idx] = (int64_t)ix;
    if (SLOT) slot_out[idx] = sx;
    if (UVW) {
        const TriV t = load_tri(tris, sx);
        double bary[3]; d3 cp;
        closest_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c), bary, &cp);
        uvw[3 * idx] = __double2float_rn(bary[0]);
        uvw[3 * idx + 1] = __double2float_rn(bary[1]);
        uvw[3 * idx + 2] = __double2float_rn(bary[2]);
    }
}

template <bool UVW, bool SLOT>
__global__ void __launch_bounds__(kQBlock) k_udf_heavy(const uint4* __restrict__ heavy,
                                                       const unsigned long long* __restrict__ n_heavy,
                                                       int64_t heavy_cap, const MeshDesc* __restrict__ meshes,
                                                       int slot_face0, const float* __restrict__ pts,
                                                       float* __restrict__ dist, int64_t* __restrict__ face_id,
                                                       float* __restrict__ uvw, int32_t* __restrict__ slot_out,
                                                       const DeviceTree tree,
                                                       unsigned long long* __restrict__ ctr) {
    __shared__ HeavyWarp shw[kQBlock / 32];
    HeavyWarp& S = shw[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t nh_all = (int64_t)*n_heavy;
    const int64_t nh = nh_all < heavy_cap ? nh_all : heavy_cap;
    while (true) {
        unsigned long long qi = 0;
        if (lane == 0) qi = atomicAdd(ctr, 1ull);
        qi = __shfl_sync(kFull, qi, 0);
        if ((int64_t)qi >= nh) break;
        const uint4 hq = heavy[qi];
        const int64_t idx = hq.x;
        int root = 0, s0 = slot_face0;
        if (meshes) {
            const MeshDesc md = meshes[hq.y];
            root = md.root;
            s0 = md.slot0;
        }
        const float3 p = load3(pts, idx);
        double bx;
        int sx, ix;
        heavy_walk(S, tree, root, p, __uint_as_float(hq.z), bx, sx, ix);
        if (lane == 0) write_nearest<UVW, SLOT>(tree.tris, idx, p, bx, sx, ix, s0, dist, face_id, uvw, slot_out);
    }
}

// -------------------------------------------------------------- few queries
// Eight lanes per query, four queries a warp, for calls with too few queries
// to make packets of near neighbours or to fill the chip with packets: lane j
// of a group tests child j of the query's node, and the leaf's triangles are
// spread over the lanes.  The walk is the query's own, nearest child first,
// so its length is a few node latencies, and the call is this one launch: no
// bucketing, no queue.  Once the walk has a bound from its first leaf and
// kFewVisits nodes behind it, a query that needs more is finished by the
// whole warp, four nodes a step (heavy_walk), as is one whose candidate list
// overflows; so few queries get a warp each, more of them two or four.
// Against unsorted packets (100 to 1,000 points on 82k faces 2.7 ms) 22 to 36
// us; 16,000 points 544 -> 111 us, sorted packets 316.  The lines:
// 32 and 96 visits are up to 1.5 and 2.5 times slower, fewer than the tree is
// deep up to 3 times; at 64k queries packets draw level (82k-face mesh 376
// against 302 us, 5,120 faces 389 against 396, 177k open tori 726 against 641).
constexpr int kFewVisits = 8;
constexpr int kFewWarps = 16;      // warps of k_udf_few on an SM at a time
constexpr int kFewCand = 32;
struct FewGroup {
    uint2 stack[kStack];           // reference, key
    uint2 cand[kFewCand];          // slot, lower bound
};
union FewWarp { FewGroup g[4]; HeavyWarp h; };
template <bool UVW, bool SLOT>
__global__ void __launch_bounds__(kQBlock) k_udf_few(int64_t n, const float* __restrict__ pts,
                                                     float* __restrict__ dist, int64_t* __restrict__ face_id,
                                                     float* __restrict__ uvw, int32_t* __restrict__ slot_out,
                                                     const DeviceTree tree, const MeshDesc* __restrict__ meshes,
                                                     const int64_t* __restrict__ qoff, int n_meshes, int slot_face0,
                                                     int per_warp) {
    __shared__ FewWarp s_few[kQBlock / 32];
    FewWarp& W = s_few[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, j = lane & 7, g = lane >> 3;
    FewGroup& S = W.g[g];
    const CTri* __restrict__ tris = tree.tris;
    const int64_t w0 = (((int64_t)blockIdx.x * kQBlock + threadIdx.x) >> 5) * per_warp;
    if (w0 >= n) return;                       // the whole warp
    const int64_t idx = w0 + g;
    const bool act = g < per_warp && idx < n;
    int root = 0, face0 = slot_face0;
    if (meshes && act) {
        int lo = 0, hi = n_meshes - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (qoff[mid] <= idx) lo = mid; else hi = mid - 1;
        }
        root = meshes[lo].root;
        face0 = meshes[lo].slot0;
    }
    const float3 p = act ? load3(pts, idx) : make_float3(0.f, 0.f, 0.f);
    const bool reach = act && isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
    float U = reach ? 1e6f : -1.f;             // bound of the squared distance (MAX_DIST^2), the group's
    int nc = 0, sp = 0, cur = root, visits = 0;
    bool live = reach, heavy = false;
    // the next entry within the bound
    auto pop = [&](float cull) {
        live = false;
        while (sp > 0) {
            const uint2 e = S.stack[--sp];
            if (__uint_as_float(e.y) <= cull) { cur = (int)e.x; live = true; break; }
        }
    };
    while (__any_sync(kFull, live)) {
        const bool inner = live && cur >= 0;
        if (__any_sync(kFull, inner)) {
            const float cull = U * 1.000002f;
            uint32_t key = kFull;
            int ref = 0;
            if (inner) {
                const float4* nb = reinterpret_cast<const float4*>(tree.wnodes + cur);
                const float4 lo = __ldg(nb + j), hi = __ldg(nb + 8 + j);
                const float d2 = box_d2(p, make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z));
                if (d2 <= cull) key = (__float_as_uint(d2) & ~7u) | (uint32_t)j;
                ref = __float_as_int(lo.w);
            }
            int pos = 0;                       // entries farther than this one
#pragma unroll
            for (int x = 1; x < 8; ++x) {
                const uint32_t k = __shfl_xor_sync(kFull, key, x);
                pos += k > key && k != kFull ? 1 : 0;
            }
            const int kept = __popc((__ballot_sync(kFull, key != kFull) >> (lane & 24)) & 0xFFu);
            if (key != kFull) S.stack[sp + pos] = make_uint2((uint32_t)ref, key & ~7u);
            __syncwarp();
            if (inner) {
                sp += kept;
                pop(cull);
                if (++visits >= kFewVisits && U < 1e6f && live) { live = false; heavy = true; }
            }
            __syncwarp();                      // the entries have been read
        }
        const bool leaf = live && cur < 0;
        if (__any_sync(kFull, leaf)) {
            float lb = 0.f, ub = CUDART_INF_F;
            int s = 0;
            bool on = false;
            if (leaf) {
                int s0, s1;
                leaf_range(cur, s0, s1);
                s = s0 + j;
                on = s < s1;
                if (on) {
                    const float4* tw = reinterpret_cast<const float4*>(tree.wtris + s);
                    float err;
                    const float d2 = tri_d2_w(p, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
                    lb = d2 - err;
                    ub = d2 + err;
                }
            }
#pragma unroll
            for (int x = 1; x < 4; x <<= 1) ub = fminf(ub, __shfl_xor_sync(kFull, ub, x));   // lanes 0 - 3 hold the leaf
            ub = __shfl_sync(kFull, ub, lane & 24);
            if (leaf) U = fminf(U, ub);
            const bool c = on && !(lb > U);    // within the bound, or undecided (no number)
            const unsigned m = (__ballot_sync(kFull, c) >> (lane & 24)) & 0xFFu;
            if (leaf) {
                const int at = nc + __popc(m & ((1u << j) - 1u));
                if (c && at < kFewCand) S.cand[at] = make_uint2((uint32_t)s, __float_as_uint(lb));
                nc += __popc(m);
                pop(U * 1.000002f);
                if (nc > kFewCand) { live = false; heavy = true; }
            }
            __syncwarp();
        }
    }
    // exact minimum (ties -> lowest face index) of the group's candidates
    double bx = CUDART_INF;
    int sx = -1, ix = INT_MAX;
    __syncwarp();
    if (!heavy) {
        for (int i = j; i < nc; i += 8) {
            const uint2 e = S.cand[i];
            if (__uint_as_float(e.y) > U) continue;
            const TriV t = load_tri(tris, (int)e.x);
            const double d = dist2_on_tri_d(to_d3(p), to_d3(t.a), to_d3(t.b), to_d3(t.c));
            if (d <= 1e6 && (d < bx || (d == bx && t.id < ix))) { bx = d; sx = (int)e.x; ix = t.id; }
        }
    }
    __syncwarp();
#pragma unroll
    for (int x = 1; x < 8; x <<= 1) {
        const double b2 = __shfl_xor_sync(kFull, bx, x);
        const int s2 = __shfl_xor_sync(kFull, sx, x), i2 = __shfl_xor_sync(kFull, ix, x);
        if (s2 >= 0 && (b2 < bx || (b2 == bx && i2 < ix))) { bx = b2; sx = s2; ix = i2; }
    }
    if (act && !heavy && j == 0) write_nearest<UVW, SLOT>(tris, idx, p, bx, sx, ix, face0, dist, face_id, uvw, slot_out);
    // the long ones, one after the other, by the whole warp
    for (unsigned hm = __ballot_sync(kFull, heavy && j == 0); hm; hm &= hm - 1u) {
        const int src = __ffs(hm) - 1;
        const float3 q = make_float3(__shfl_sync(kFull, p.x, src), __shfl_sync(kFull, p.y, src), __shfl_sync(kFull, p.z, src));
        const float u = __shfl_sync(kFull, U, src);
        const int r = __shfl_sync(kFull, root, src), f0 = __shfl_sync(kFull, face0, src);
        heavy_walk(W.h, tree, r, q, u, bx, sx, ix);
        if (lane == 0) write_nearest<UVW, SLOT>(tris, w0 + (src >> 3), q, bx, sx, ix, f0, dist, face_id, uvw, slot_out);
    }
}

// ------------------------------------------------------------ watertight
// A triangle whose FP32 upper bound of the squared distance is below this is in
// the normal sum; only those near the radius are settled in double.  The bound
// needs the slack (cp rounded to float moves the distance by less) to stay
// below 1e-6 itself, so no coordinate above 1e3 takes this way.  A closest
// point on a vertex has six or more members, whose double tests were a quarter
// of the sign pass (8.4M points on 82k faces: 5.21 -> 4.89 ms a call; with the
// list's triangles tested on their frames, tri_d2_w, 4.68).
constexpr float kInSum = 0.999999e-6f;
// Sum of unit normals of every triangle whose squared distance to cp is
// below 1e-6 (src/bvh.cu:356-396; the division by the count does not change
// the sign and is omitted).  cp lies on the triangle in soup slot `own` (the
// query's nearest), so that one needs no distance test.
__device__ d3 normal_sum(const CNode* __restrict__ nodes, const CTri* __restrict__ tris, d3 cp, int root, int own) {
    const float3 cf = make_float3(__double2float_rn(cp.x), __double2float_rn(cp.y), __double2float_rn(cp.z));
    const float cinf = f3inf(cf);
    const float r = 1e-3f + 4e-7f * (1.f + cinf);
    const float r2 = r * r * 1.00001f;
    const float slack = 1e-9f * (1.f + cinf);
    d3 sum{0.0, 0.0, 0.0};
    int st[kStack];
    int sp = 0;
    st[sp++] = root;
    while (sp > 0) {
        const int ref = st[--sp];
        if (ref >= 0) {
            const NodeView nd = load_node(nodes, ref);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t m = meta_of(nd, j);
                float3 lo, hi;
                child_box(nd, j, lo, hi);
                if (m != kEmpty && box_d2(cf, lo, hi) <= r2) st[sp++] = child_ref(nd, m);
            }
        } else {
            int s0, s1;
            leaf_range(ref, s0, s1);
            for (int s = s0; s < s1; ++s) {
                const TriV t = load_tri(tris, s);
                float err;
                const float d2 = tri_d2_f(cf, t, &err);
                if (d2 - err - slack > 1.000001e-6f) continue;
                double bary[3]; d3 q;
                const d3 a = to_d3(t.a), b = to_d3(t.b), c = to_d3(t.c);
                if (s == own || d2 + err + slack < kInSum || closest_on_tri_d(cp, a, b, c, bary, &q) < 1e-6) {
                    const d3 nr = dcross(dsub(b, a), dsub(c, a));
                    const double len = __dsqrt_rn(ddot(nr, nr));
                    if (len > 0.0) sum = dadd(sum, d3{dD(nr.x, len), dD(nr.y, len), dD(nr.z, len)});
                }
            }
        }
    }
    return sum;
}

// normal_sum over a precomputed candidate list of cp's triangle (k_near_lists):
// the same tests in the same order, without the walk from the root, and the
// unit normals read from the table k_near_lists computed them into (the same
// operations as normal_sum's).
__device__ d3 normal_sum_list(const CTri* __restrict__ tris, const WTri* __restrict__ wtris, d3 cp, int own, const int32_t* __restrict__ lst,
                              int count, const double* __restrict__ nrm) {
    const float3 cf = make_float3(__double2float_rn(cp.x), __double2float_rn(cp.y), __double2float_rn(cp.z));
    const float slack = 1e-9f * (1.f + f3inf(cf));
    d3 sum{0.0, 0.0, 0.0};
    for (int k = 0; k < count; ++k) {
        const int s = __ldg(lst + k);
        const float4* tw = reinterpret_cast<const float4*>(wtris + s);
        float err;
        const float d2 = tri_d2_w(cf, make_triw(__ldg(tw), __ldg(tw + 1), __ldg(tw + 2), __ldg(tw + 3)), &err);
        if (d2 - err - slack > 1.000001e-6f) continue;
        bool in = s == own || d2 + err + slack < kInSum;
        if (!in) {
            const TriV t = load_tri(tris, s);
            in = dist2_on_tri_d(cp, to_d3(t.a), to_d3(t.b), to_d3(t.c)) < 1e-6;
        }
        if (in)
            // a zero normal (degenerate triangle) leaves the sum unchanged: its
            // components are never -0, so adding +0 is exact
            sum = dadd(sum, d3{__ldg(nrm + 3 * s), __ldg(nrm + 3 * s + 1), __ldg(nrm + 3 * s + 2)});
    }
    return sum;
}

// True when an axis among the two triangles' normals and the nine cross
// products of their edges separates a and b by more than r: then no point of
// b lies within r of a point of a.  Any axis u is a valid separating axis, so
// rounding in u itself is harmless; each projection onto u is off by at most
// a few ulps of |u| max|v|, covered by the margin 2e-6 (1 + scale) |u| added to
// r (scale: the larger max |coordinate| of the two triangles).  Degenerate
// axes (|u| = 0) separate nothing.
__device__ bool tri_gap_exceeds(const TriV& a, const TriV& b, float r, float scale) {
    const float3 ea[3] = {f3sub(a.b, a.a), f3sub(a.c, a.b), f3sub(a.a, a.c)};
    const float3 eb[3] = {f3sub(b.b, b.a), f3sub(b.c, b.b), f3sub(b.a, b.c)};
    const float rr = r + 2e-6f * (1.f + scale);
    auto sep = [&](float3 u) {
        const float l2 = f3dot(u, u);
        if (!(l2 > 0.f)) return false;
        const float a0 = f3dot(u, a.a), a1 = f3dot(u, a.b), a2 = f3dot(u, a.c);
        const float b0 = f3dot(u, b.a), b1 = f3dot(u, b.b), b2 = f3dot(u, b.c);
        const float amin = fminf(a0, fminf(a1, a2)), amax = fmaxf(a0, fmaxf(a1, a2));
        const float bmin = fminf(b0, fminf(b1, b2)), bmax = fmaxf(b0, fmaxf(b1, b2));
        return fmaxf(bmin - amax, amin - bmax) > rr * 1.0001f * sqrtf(l2);
    };
    if (sep(f3cross(ea[0], ea[1])) || sep(f3cross(eb[0], eb[1]))) return true;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (sep(f3cross(ea[i], eb[j]))) return true;
    return false;
}

// Candidate lists of the watertight normal sum.  For soup slot t: every slot
// whose triangle's bounding box meets t's box grown by r = 1.001e-3 + 1e-6 (1 +
// max |coordinate|) and that no separating axis (tri_gap_exceeds) puts more
// than r from t, in the order normal_sum's walk reaches them (depth-first,
// children in the same push order, slots ascending in a leaf).  A point cp on
// triangle t has every triangle within normal_sum's radius of it on t's list
// (the radius is at most 1e-3 + 4e-7 (1 + |cp|_inf) and |cp| <= max |vertex|),
// so the list replaces the walk and keeps the summation order.  cnt[t] = -1
// when more than kNear slots qualify: that query walks the tree.
__global__ void __launch_bounds__(kQBlock) k_near_lists(int64_t nt, const CNode* __restrict__ nodes,
                                                        const CTri* __restrict__ tris, int root,
                                                        int32_t* __restrict__ cnt, int32_t* __restrict__ lst,
                                                        double* __restrict__ nrm, int* __restrict__ any_ovf) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += (int64_t)gridDim.x * blockDim.x) {
        const TriV a = load_tri(tris, (int)t);
        {
            const d3 da = to_d3(a.a), db = to_d3(a.b), dc = to_d3(a.c);
            const d3 nr = dcross(dsub(db, da), dsub(dc, da));
            const double len = __dsqrt_rn(ddot(nr, nr));
            const bool ok = len > 0.0;
            nrm[3 * t] = ok ? dD(nr.x, len) : 0.0;
            nrm[3 * t + 1] = ok ? dD(nr.y, len) : 0.0;
            nrm[3 * t + 2] = ok ? dD(nr.z, len) : 0.0;
        }
        float3 lo = make_float3(fminf(a.a.x, fminf(a.b.x, a.c.x)), fminf(a.a.y, fminf(a.b.y, a.c.y)),
                                fminf(a.a.z, fminf(a.b.z, a.c.z)));
        float3 hi = make_float3(fmaxf(a.a.x, fmaxf(a.b.x, a.c.x)), fmaxf(a.a.y, fmaxf(a.b.y, a.c.y)),
                                fmaxf(a.a.z, fmaxf(a.b.z, a.c.z)));
        const float vinf = fmaxf(f3inf(lo), f3inf(hi));
        const float r = 1.001e-3f + 1e-6f * (1.f + vinf);
        lo = make_float3(lo.x - r, lo.y - r, lo.z - r);
        hi = make_float3(hi.x + r, hi.y + r, hi.z + r);
        int32_t* out = lst + t * kNear;
        int c = 0;
        int st[kStack];
        int sp = 0;
        st[sp++] = root;
        while (sp > 0) {
            const int ref = st[--sp];
            if (ref >= 0) {
                const NodeView nd = load_node(nodes, ref);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t m = meta_of(nd, j);
                    float3 clo, chi;
                    child_box(nd, j, clo, chi);
                    if (m != kEmpty && clo.x <= hi.x && clo.y <= hi.y && clo.z <= hi.z && chi.x >= lo.x &&
                        chi.y >= lo.y && chi.z >= lo.z)
                        st[sp++] = child_ref(nd, m);
                }
            } else {
                int s0, s1;
                leaf_range(ref, s0, s1);
                for (int s = s0; s < s1; ++s) {
                    const TriV b = load_tri(tris, s);
                    if (fminf(b.a.x, fminf(b.b.x, b.c.x)) <= hi.x && fminf(b.a.y, fminf(b.b.y, b.c.y)) <= hi.y &&
                        fminf(b.a.z, fminf(b.b.z, b.c.z)) <= hi.z && fmaxf(b.a.x, fmaxf(b.b.x, b.c.x)) >= lo.x &&
                        fmaxf(b.a.y, fmaxf(b.b.y, b.c.y)) >= lo.y && fmaxf(b.a.z, fmaxf(b.b.z, b.c.z)) >= lo.z &&
                        (s == (int)t ||
                         !tri_gap_exceeds(a, b, r, fmaxf(vinf, fmaxf(f3inf(b.a), fmaxf(f3inf(b.b), f3inf(b.c))))))) {
                        if (c < kNear) out[c] = s;
                        ++c;
                    }
                }
            }
        }
        cnt[t] = c <= kNear ? c : -1;
        if (c > kNear) atomicOr(any_ovf, 1);
    }
}

// Watertight sign: copysign(distance, normal_sum . (p - cp)), cp the closest
// point of the query's nearest triangle (soup slot `own`).  LIST: the normal
// sum over own's candidate list; a query whose list overflowed is queued in
// ovf for k_sign_watertight_ovf (single BVH).  !LIST: the walk (arenas).
constexpr int kSignBlocks = 5;   // blocks per SM (8.4M points, whole call: 4 4.81 ms, 5 4.68, 6 4.72)
template <bool LIST>
__global__ void __launch_bounds__(kQBlock, LIST ? kSignBlocks : 1)
k_sign_watertight(Work w, const uint32_t* __restrict__ order, const float* __restrict__ pts, float* __restrict__ dist,
                  const int32_t* __restrict__ slots, const CNode* __restrict__ nodes, const CTri* __restrict__ tris,
                  const WTri* __restrict__ wtris, const NearLists near, uint32_t* __restrict__ ovf, unsigned long long* __restrict__ ovf_n,
                  unsigned long long* __restrict__ ctr, int64_t grab, int block_grabs) {
    __shared__ int s_left;
    if (block_grabs > 0) {
        if (threadIdx.x == 0) s_left = block_grabs;
        __syncthreads();
    }
    PacketQueue pq(ctr, w.packets(), grab, block_grabs > 0 ? &s_left : nullptr);
    for (int64_t pk = pq.take(); pk >= 0; pk = pq.take()) {
        int64_t start, qoff;
        int cnt, root, s0;
        w.get(pk, start, cnt, root, s0, qoff);
        if ((int)(threadIdx.x & 31) >= cnt) continue;
        const int64_t q = start + (threadIdx.x & 31);
        const int64_t idx = order ? (int64_t)order[q] : q;
        const int own = slots[idx];
        const int nc = LIST ? __ldg(near.cnt + own) : -1;  // in flight during the closest point
        const d3 pd = to_d3(load3(pts, idx));
        const TriV t = load_tri(tris, own);
        double bary[3]; d3 cp;
        closest_on_tri_d(pd, to_d3(t.a), to_d3(t.b), to_d3(t.c), bary, &cp);
        if (LIST && nc < 0) {
            ovf[atomicAdd(ovf_n, 1ull)] = (uint32_t)idx;
            continue;
        }
        const d3 ns = LIST ? normal_sum_list(tris, wtris, cp, own, near.lst + (int64_t)own * kNear, nc, near.nrm)
                           : normal_sum(nodes, tris, cp, root, own);
        // copysign(distance, avg_normal . (p - cp))
        const double s = ddot(ns, dsub(pd, cp));
        const float d = dist[idx];
        dist[idx] = signbit(s) ? -d : d;
    }
}
// The queries k_sign_watertight<true> queued (their lists overflowed): the
// walk from root 0.
__global__ void __launch_bounds__(kQBlock) k_sign_watertight_ovf(const uint32_t* __restrict__ ovf,
                                                                 const unsigned long long* __restrict__ ovf_n,
                                                                 const float* __restrict__ pts,
                                                                 float* __restrict__ dist,
                                                                 const int32_t* __restrict__ slots,
                                                                 const CNode* __restrict__ nodes,
                                                                 const CTri* __restrict__ tris) {
    const int64_t n = (int64_t)*ovf_n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t idx = ovf[i];
        const int own = slots[idx];
        const d3 pd = to_d3(load3(pts, idx));
        const TriV t = load_tri(tris, own);
        double bary[3]; d3 cp;
        closest_on_tri_d(pd, to_d3(t.a), to_d3(t.b), to_d3(t.c), bary, &cp);
        const d3 ns = normal_sum(nodes, tris, cp, 0, own);
        const double s = ddot(ns, dsub(pd, cp));
        const float d = dist[idx];
        dist[idx] = signbit(s) ? -d : d;
    }
}

// --------------------------------------------------------------- raystab
// Negative iff all 64 stab rays (for k = 0..31: -d_k, then +d_k) hit the mesh
// within [0, 1000) (src/bvh.cu:408-427); the first miss ends the query.
// Whether all rays hit does not depend on the order they are traced in.
//
// Closed meshes.  Where every edge of a mesh bounds an even number of its
// triangles (k_edge_parity), the mesh is a cycle modulo two: along any ray
// from a point that meets no edge, the number of crossings has the parity of
// the point's winding number.  So when the crossings of one stab ray, all
// certain by the FP32 test's error bounds, are odd in number, every ray from
// the point crosses the mesh and all 64 hit: the point is inside after one
// ray.  No crossing means outside; an even number, an undecided triangle, a
// mesh that is not closed, or a point so far away that a crossing could lie
// past t = 1000 leave the query to its other rays.  (A stab ray that the
// rounding of the double test lets slip between two triangles at their common
// edge, about 1e-14 of all rays, is not seen this way.)  Inside points took
// 64 rays, bound by divergence (12.5 of 32 lanes): 2.1M points in the box of a
// closed 82k-face mesh, 18.9 -> 4.2 ms with the faster distance search.

// Hash of an undirected edge by its end points' coordinates (0 for an edge
// of no length): mesh edges cancel in pairs under XOR.  mix64 is David
// Stafford's Mix01, a variant of MurmurHash3's 64-bit finaliser.
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 31;
    x *= 0x7fb5d329728ea185ull;
    x ^= x >> 27;
    x *= 0x81dadef4bc2dd44dull;
    return x ^ (x >> 33);
}
__device__ __forceinline__ unsigned long long point_hash(float3 v) {   // -0 counts as 0
    const unsigned long long x = __float_as_uint(v.x + 0.f), y = __float_as_uint(v.y + 0.f), z = __float_as_uint(v.z + 0.f);
    return mix64(mix64(x | (y << 32)) + z + 0x9e3779b97f4a7c15ull);
}
__device__ __forceinline__ unsigned long long edge_hash(unsigned long long a, unsigned long long b) {
    if (a == b) return 0ull;
    const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
    return mix64(mix64(lo) + 3ull * hi + 1ull);
}
// XOR of the edge hashes of every mesh's triangles into parity[m], zeroed
// before.  Mesh m has the faces face_off[m] .. face_off[m + 1] - 1, face i the
// soup slot face_slot[i] (both null: one mesh, every slot of nt).  The result is 0
// for a closed mesh, and for another one with probability 2^-64.  It runs with each raystab call (82k triangles: 3 us)
// rather than once per tree, so there is no state to keep right across
// refits, streams and captures.
__global__ void __launch_bounds__(256) k_edge_parity(int64_t nt, const CTri* __restrict__ tris,
                                                     const int64_t* __restrict__ face_off,
                                                     const int32_t* __restrict__ face_slot, int M,
                                                     unsigned long long* __restrict__ parity) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned long long h = 0ull;
    int mesh = -1;
    for (int k = 0; k < 4; ++k) {   // 128 consecutive faces a warp
        const int64_t s = warp * 128 + 32 * k + lane;
        int m = mesh;
        unsigned long long e = 0ull;
        if (s < nt) {
            const TriV t = load_tri(tris, face_slot ? face_slot[s] : (int)s);
            const unsigned long long a = point_hash(t.a), b = point_hash(t.b), c = point_hash(t.c);
            e = edge_hash(a, b) ^ edge_hash(b, c) ^ edge_hash(c, a);
            m = 0;
            if (face_off) {
                int lo = 0, hi = M - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (face_off[mid] <= s) lo = mid; else hi = mid - 1;
                }
                m = lo;
            }
        }
        if (m != mesh && mesh >= 0) { atomicXor(&parity[mesh], h); h = 0ull; }
        mesh = m;
        h ^= e;
    }
    const int m0 = __shfl_sync(kFull, mesh, 0);
    if (__all_sync(kFull, mesh == m0 || mesh < 0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) h ^= __shfl_xor_sync(kFull, h, o);
        if (lane == 0 && m0 >= 0) atomicXor(&parity[m0], h);
    } else if (mesh >= 0) {
        atomicXor(&parity[mesh], h);
    }
}

// First raystab pass: each lane traces one query's first stab line, ray 0 =
// -d_0 and, when that hits (or its count decides nothing), ray 1 = +d_0.  A
// query whose rays both hit is appended to `cand` (query index, stab offset,
// root: warp-aggregated atomic on cand_n), for k_sign_raystab_lines.  Outside
// points mostly see a ray miss and end in this pass, as do the inside points
// of closed meshes; the candidates are mostly inside points of other meshes,
// which need every ray.
//
// Work is per lane, as in k_ray_lanes: a warp takes a chunk of packets (queries
// in Morton-cell order), prepares its queries in lockstep (position, stab
// offset, d_0, root, whether ray 0 counts crossings), and hands them to lanes
// whenever kStabRefill are idle; its lanes stay on the same kind of step, inner
// nodes until few are at one, then leaves.  Lanes refilled one by one, each on
// its own step, took 2.2 of the 4.1 ms of 2.1M points on a closed 82k-face
// mesh; in batches the call takes 3.0 (refill at 12 and 20 idle lanes 3.2 and 3.5).
constexpr int kChunkMax = 2;      // packets per raystab chunk
constexpr int kStabRefill = 6;   // idle lanes that take new queries
constexpr int kStabInner = 12;    // fewer lanes at inner nodes than this wait for those at leaves
constexpr int kStabBlocks = 6;    // blocks per SM
struct StabQuery { float px, py, pz, dx, dy, dz, ox, oy; uint32_t idx; int root; };   // d_0, stab offset; root -1: none, -2 - root: counting
__global__ void __launch_bounds__(kQBlock, kStabBlocks) k_sign_raystab(Work w, const uint32_t* __restrict__ order,
                                                          const float* __restrict__ pts, float* __restrict__ dist,
                                                          const CNode* __restrict__ nodes,
                                                          const CTri* __restrict__ tris,
                                                          unsigned long long* __restrict__ ctr, int64_t grab,
                                                          uint4* __restrict__ cand,
                                                          unsigned long long* __restrict__ cand_n,
                                                          const unsigned long long* __restrict__ parity) {
    __shared__ StabQuery s_q[kQBlock / 32][kChunkMax * 32];
    StabQuery* sq = s_q[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const float tmaxf = 1000.0f;
    const float cull = cull_of(1000.0);
    PacketQueue pq(ctr, w.packets(), grab);
    int next = 0, total = 0;                 // the chunk's queries: next to hand out, number
    bool more = true;                        // more chunks may come
    bool live = false, second = false, counting = false, unsure = false, any = false, degen = false;
    int crossings = 0, root = 0, cur = 0, sp = 0;
    int64_t idx = -1;
    float3 p = make_float3(0.f, 0.f, 0.f), d = p, inv = p;
    float2 off = make_float2(0.f, 0.f);
    float dinf = 0.f;
    int st[kStack];
    auto start_ray = [&]() {
        inv = ray_inv_approx(d);
        degen = ray_degenerate(inv);
        dinf = f3inf(d);
        sp = 0;
        cur = root;
    };
    while (true) {
        const unsigned idle = __ballot_sync(kFull, !live);
        if (idle == kFull || ((more || next < total) && __popc(idle) >= kStabRefill)) {
            if (next >= total && more) {     // the next chunk
                int64_t pk0, pk1;
                more = pq.take_range(pk0, pk1);
                total = more ? (int)(pk1 - pk0) * 32 : 0;
                next = 0;
                __syncwarp();                // the last chunk's queries have been read
                for (int i = lane; i < total; i += 32) {
                    int64_t start, qoff;
                    int cnt, rt, s0;
                    w.get(pk0 + (i >> 5), start, cnt, rt, s0, qoff);
                    StabQuery q;
                    q.root = -1;
                    if ((i & 31) < cnt) {
                        const int64_t qi = start + (i & 31);
                        const int64_t id = order ? (int64_t)order[qi] : qi;
                        // the stab stream of a query is its index within its own call / mesh
                        const float2 o2 = stab_offset((uint32_t)(id - qoff));
                        const float3 v = load3(pts, id), sd = stab_dir(0, o2);
                        // closed, and the whole root box within t < 1000 of the point
                        const CNode* rn = nodes + rt;
                        float far2 = 0.f;
                        const float lo[3] = {rn->ox, rn->oy, rn->oz}, qc[3] = {v.x, v.y, v.z};
                        const int ex[3] = {rn->ex, rn->ey, rn->ez};
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const float f = fmaxf(fabsf(lo[k] - qc[k]), fabsf(fmaf(255.f, exp2i(ex[k]), lo[k]) - qc[k]));
                            far2 = fmaf(f, f, far2);
                        }
                        const bool count = parity[w.mesh_of(pk0 + (i >> 5))] == 0ull && far2 < 9.8e5f;
                        q = StabQuery{v.x, v.y, v.z, sd.x, sd.y, sd.z, o2.x, o2.y, (uint32_t)id, count ? -2 - rt : rt};
                    }
                    sq[i] = q;
                }
                __syncwarp();
            }
            if (next < total) {
                const int k = next + __popc(idle & lt);
                if (!live && k < total && sq[k].root != -1) {
                    const StabQuery q = sq[k];
                    counting = q.root < 0;
                    root = counting ? -2 - q.root : q.root;
                    idx = q.idx;
                    p = make_float3(q.px, q.py, q.pz);
                    d = make_float3(-q.dx, -q.dy, -q.dz);
                    off = make_float2(q.ox, q.oy);
                    second = unsure = any = false;
                    crossings = 0;
                    live = true;
                    start_ray();
                }
                next += __popc(idle);
            } else if (idle == kFull && !more) {
                break;
            }
            continue;
        }
        bool ended = false, hit = false;
        // inner nodes
        while (true) {
            const bool inner = live && !ended && cur >= 0;
            const unsigned in = __ballot_sync(kFull, inner);
            if (!in || (__popc(in) < kStabInner && __any_sync(kFull, live && !ended && cur < 0))) break;
            if (inner) {
                const NodeView nd = load_node(nodes, cur);
                if (degen) push_ray_children(nd, p, inv, cull, st, sp);
                else push_ray_children_affine(nd, p, inv, cull, st, sp);
                if (sp > 0) cur = st[--sp];
                else ended = true;
            }
            if (__popc(__ballot_sync(kFull, !live || ended)) >= kStabRefill) break;
        }
        // leaves
        if (live && !ended && cur < 0) {
            int a, b;
            leaf_range(cur, a, b);
            for (int s = a; s < b && !hit; ++s) {
                const TriV t = load_tri(tris, s);
                float tt, terr;
                const int c = ray_tri_f(p, d, dinf, t, tmaxf, &tt, &terr);
                bool on = c == 1;
                if (c < 0) {
                    double t64;
                    on = ray_tri_d(to_d3(p), to_d3(d), to_d3(t.a), to_d3(t.b), to_d3(t.c), 1000.0, &t64);
                    unsure = true;
                }
                any |= on;
                crossings += on ? 1 : 0;
                hit = on && !counting;
            }
            if (!hit) {
                if (sp > 0) cur = st[--sp];
                else ended = true;
            }
        }
        __syncwarp();
        // rays that came to their end
        if (ended) {
            if (counting && any && (unsure || !(crossings & 1))) hit = true;   // ray 0 hits, no more is known
            else {
                if (counting && any) dist[idx] = -dist[idx];                   // inside: every ray hits
                live = false;                                                  // else a ray missed: outside
            }
            counting = false;
        }
        if (hit) {
            if (!second) {
                second = true;
                d = make_float3(-d.x, -d.y, -d.z);
                start_ray();
            } else {
                const cooperative_groups::coalesced_group g = cooperative_groups::coalesced_threads();
                unsigned long long b = 0;
                if (g.thread_rank() == 0) b = atomicAdd(cand_n, (unsigned long long)g.size());
                b = g.shfl(b, 0) + g.thread_rank();
                cand[b] = make_uint4((uint32_t)idx, __float_as_uint(off.x), __float_as_uint(off.y), (uint32_t)root);
                live = false;
            }
        }
        __syncwarp();
    }
}

// Second raystab pass: a warp per candidate query.  The query's rays
// first_ray .. 63 (ray 2k = -d_k, ray 2k + 1 = +d_k, all from the query
// point; the first pass traced the others) form a pool: lane l starts with
// ray first_ray + l and, whenever its ray hits, takes the next ray of the
// pool, so lanes stay busy until the pool is empty.  A ray that finds no hit
// ends the query for the whole warp (__any_sync): the point is outside; when
// the pool is empty and every lane's ray has hit, it is inside.  Each step
// of a lane is one inner node or one triangle, so lanes at inner nodes and
// lanes at leaves run steps of similar length side by side.  The rays of a
// warp start at the same point, so the first levels of their walks read the
// same nodes.  Warps take candidates from a counter in the order the first
// pass appended them (near one another in space).
__global__ void __launch_bounds__(kQBlock, 10) k_sign_raystab_lines(const float* __restrict__ pts,
                                                                float* __restrict__ dist,
                                                                const CNode* __restrict__ nodes,
                                                                const CTri* __restrict__ tris,
                                                                const uint4* __restrict__ cand,
                                                                const unsigned long long* __restrict__ cand_n,
                                                                unsigned long long* __restrict__ next, int first_ray) {
    __shared__ int s_pool[kQBlock / 32];
    __shared__ float3 s_dir[kQBlock / 32][32];   // the query's stab directions d_0 .. d_31
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned long long n = *cand_n;
    const float tmaxf = 1000.0f;
    const float cull = cull_of(1000.0);
    int st[kStack];
    while (true) {
        unsigned long long c = 0;
        if (lane == 0) c = atomicAdd(next, 1ull);
        c = __shfl_sync(kFull, c, 0);
        if (c >= n) break;
        const uint4 e = cand[c];
        const int64_t idx = e.x;
        const float2 off = make_float2(__uint_as_float(e.y), __uint_as_float(e.z));
        const int root = (int)e.w;
        const float3 p = load3(pts, idx);
        if (lane == 0) s_pool[wib] = first_ray + 32;
        s_dir[wib][lane] = stab_dir((uint32_t)lane, off);   // lane k: direction k
        __syncwarp();
        int ray = first_ray + lane;            // >= 64: this lane has no ray left
        float3 d = make_float3(0.f, 0.f, 0.f), inv = d;
        bool degen = false;
        float dinf = 0.f;
        int sp = 0, ls = 0, le = 0;            // stack; triangles [ls, le) of the current leaf
        auto start_ray = [&]() {
            const float3 sd = s_dir[wib][ray >> 1];
            d = (ray & 1) ? sd : make_float3(-sd.x, -sd.y, -sd.z);
            inv = ray_inv_approx(d);
            degen = ray_degenerate(inv);
            dinf = f3inf(d);
            sp = 0;
            st[sp++] = root;
            ls = le = 0;
        };
        if (ray < 64) start_ray();
        bool inside = false;
        while (true) {
            bool miss = false;
            if (ray < 64) {
                bool hit = false;
                if (ls >= le) {
                    if (sp == 0) {
                        miss = true;
                    } else {
                        const int ref = st[--sp];
                        if (ref >= 0) {
                            const NodeView nd = load_node(nodes, ref);
                            if (degen) push_ray_children(nd, p, inv, cull, st, sp);
                            else push_ray_children_affine(nd, p, inv, cull, st, sp);
                        } else {
                            leaf_range(ref, ls, le);
                        }
                    }
                }
                if (ls < le) {                 // one triangle of the current leaf
                    const TriV t = load_tri(tris, ls++);
                    float tt, terr;
                    const int cl = ray_tri_f(p, d, dinf, t, tmaxf, &tt, &terr);
                    if (cl == 1) hit = true;
                    else if (cl < 0) {
                        double t64;
                        hit = ray_tri_d(to_d3(p), to_d3(d), to_d3(t.a), to_d3(t.b), to_d3(t.c), 1000.0, &t64);
                    }
                }
                if (hit) {
                    ray = atomicAdd(&s_pool[wib], 1);
                    if (ray < 64) start_ray();
                }
            }
            if (__any_sync(kFull, miss)) break;            // a stab ray left the mesh: outside
            if (__all_sync(kFull, ray >= 64)) { inside = true; break; }
        }
        if (inside && lane == 0) dist[idx] = -dist[idx];
        __syncwarp();
    }
}

// ---------------------------------------------------------------- rays
constexpr int kUnit = 8;   // rays per unit of the ray packet order (k_ray_order), 4 units per packet
// Ray of `lane` in packet pk: the unit lane / 8 of the packet's four entries
// of order[] (units of 8 consecutive rays); n when there is none.
__device__ __forceinline__ int64_t packet_ray(int64_t pk, int lane, int64_t n, const uint32_t* __restrict__ order) {
    const int64_t units = (n + kUnit - 1) / kUnit;
    const int64_t slot = pk * (32 / kUnit) + lane / kUnit;
    return slot < units ? (int64_t)__ldg(order + slot) * kUnit + lane % kUnit : n;
}
// Whether a window's packets (k_ray_order) are traced as packets (k_ray) or ray
// by ray (k_ray_lanes).  k_ray bounds a unit's rays by intervals, which keep
// ever more nodes that no ray needs as the unit spreads against the faces it
// meets, so a packet is within limits when
//  - each unit's rays are all but parallel (unit directions within kCohDir,
//    max-norm: half a degree; and, at the distance of the mesh, within kCohFaces
//    faces, the extent of the root box over the square root of their number),
//  - its units are nearly so (kCohUnits),
//  - and they start close together (origins within kCohOrigin of the extent).
// The packets of a window go one way, packets if half of them are within
// limits, so that one kernel's longest walks do not follow the other's; only
// packets beyond twice the limits are always traced ray by ray.  A call of few
// rays, which fills the chip with neither, is bound by its longest walk, the
// longer one in a packet: a quarter of the limits (kCohFew).
//
// 1M camera rays with directions jittered by 0, 0.001, 0.002, 0.004 radians
// against no density limit and a decision per packet: 1.3M faces 0.68, 0.82,
// 0.84, 0.84 against 0.67, 1.23, 1.97, 3.35 ms, 82k faces 0.20, 0.26, 0.34, 0.36
// against 0.20, 0.30, 0.40, 0.59; 0.26M camera rays on 1.3M faces 0.41 against
// 0.70.  kCohFaces 2 / 2.5 / 5: 0.82 / 0.68 / 0.68, 0.82 / 0.82 / 1.08 ms at 0 and
// 0.001.  33.5M exact camera rays 3.14 against 3.14, at kCohDir 0.005 3.2.
// 65k of them, 0.0009 radians apart, on 1.3M faces 0.18 against 0.34 ms without
// kCohFew, 0.0002 apart 0.12 as packets and 0.14 ray by ray.
constexpr float kCohDir = 0.008f;
constexpr float kCohFaces = 3.f;
constexpr float kCohUnits = 0.03f;
constexpr float kCohOrigin = 0.01f;
constexpr int64_t kFewRays = 1 << 17;
constexpr float kCohFew = 0.25f;
// A direction component up to kParallel of the ray's largest, or up to this,
// counts as parallel to the planes of its axis (kind 2 below), whatever its
// sign.  A ray whose origin lies in a box's plane does
// not leave the box there when the component is zero, nor, as far as the double
// test can tell (its own rounding is about 1e-16 of the origin's distance), when
// it is that small; below 1e-30 its reciprocal would not stay a number.
constexpr float kSmallest = 1e-30f;
// One axis of the node tests of a lane's eight rays, in two halves of four
// (a pair of values each): what the halves' origins lie within and their
// directions' reciprocals.  kind: 0 all directions positive, 1 all negative, 2
// otherwise: signs that differ, or a ray parallel to the axis' planes, which
// is between them for every parameter or for none.
struct RayAxis { f2 on, of, i0, i1; int kind; };
// The axis of the lane's quad of rays and the other quad of its group of
// eight, from o, d of the lane's ray (ok: the lane has one); dinf: the ray's
// largest component.
__device__ __forceinline__ RayAxis ray_axis(float o, float d, float dinf, bool ok) {
    float o0 = ok ? o : CUDART_INF_F, o1 = ok ? o : -CUDART_INF_F;
    float d0 = ok ? d : CUDART_INF_F, d1 = ok ? d : -CUDART_INF_F;
#pragma unroll
    for (int s = 1; s < 4; s <<= 1) {
        o0 = fminf(o0, __shfl_xor_sync(kFull, o0, s));
        o1 = fmaxf(o1, __shfl_xor_sync(kFull, o1, s));
        d0 = fminf(d0, __shfl_xor_sync(kFull, d0, s));
        d1 = fmaxf(d1, __shfl_xor_sync(kFull, d1, s));
    }
    const float along = fmaxf(kParallel * dinf, kSmallest);
    const unsigned group = 0xFFu << (threadIdx.x & 24);
    const bool up = (~__ballot_sync(kFull, !ok || d > along) & group) == 0u;
    const bool down = (~__ballot_sync(kFull, !ok || d < -along) & group) == 0u;
    RayAxis r;
    r.kind = up ? 0 : (down ? 1 : 2);
    float on, of, i0, i1;
    if (r.kind == 2) {   // reached upwards from o1 by the largest direction, downwards from o0 by the smallest
        on = o1; of = o0;
        i0 = d1 > kSmallest ? 1.0f / d1 : 1.0f / kSmallest;
        i1 = d0 < -kSmallest ? 1.0f / d0 : -1.0f / kSmallest;
    } else {
        on = r.kind == 0 ? o1 : o0;
        of = r.kind == 0 ? o0 : o1;
        i0 = 1.0f / d0;
        i1 = 1.0f / d1;
    }
    r.on = f2pack(-on, -__shfl_xor_sync(kFull, on, 4));   // negated
    r.of = f2pack(-of, -__shfl_xor_sync(kFull, of, 4));
    r.i0 = f2pack(i0, __shfl_xor_sync(kFull, i0, 4));
    r.i1 = f2pack(i1, __shfl_xor_sync(kFull, i1, 4));
    return r;
}
// Bounds of the parameter at which rays of either half lie between the box
// planes lo and hi of the axis: no ray enters before tn or leaves after tf.
// MIXED: kind 2 may occur.
template <bool MIXED>
__device__ __forceinline__ void axis_slab(const RayAxis& r, float lo, float hi, float tn[2], float tf[2]) {
    const bool neg = r.kind == 1;
    const float near = neg ? hi : lo, far = neg ? lo : hi;
    const f2 A = f2add(f2pack(near, near), r.on), B = f2add(f2pack(far, far), r.of);
    float p[2], q[2], u[2], v[2];
    f2unpack(f2mul(A, r.i0), p[0], p[1]);
    f2unpack(f2mul(A, r.i1), q[0], q[1]);
    f2unpack(f2mul(B, r.i0), u[0], u[1]);
    f2unpack(f2mul(B, r.i1), v[0], v[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        tn[h] = fminf(p[h], q[h]);
        tf[h] = fmaxf(u[h], v[h]);
        if (MIXED && r.kind == 2) { tn[h] = fmaxf(p[h], v[h]); tf[h] = CUDART_INF_F; }
    }
}
// Entry bound (ordered bits of max(tn, 0)) of the lane's eight rays into the
// box, kFull when no half needs it within its bound c[h].  As in box_ray the
// bounds are widened by 1e-6 relative for their roundings, here by products
// that keep infinities: an unused child has tn = inf, tf = -inf.
template <bool MIXED>
__device__ __forceinline__ uint32_t group_entry(const RayAxis& X, const RayAxis& Y, const RayAxis& Z, float4 lo,
                                                float4 hi, const float c[2]) {
    float xn[2], xf[2], yn[2], yf[2], zn[2], zf[2];
    axis_slab<MIXED>(X, lo.x, hi.x, xn, xf);
    axis_slab<MIXED>(Y, lo.y, hi.y, yn, yf);
    axis_slab<MIXED>(Z, lo.z, hi.z, zn, zf);
    uint32_t key = kFull;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float tn = fmaxf(max3(xn[h], yn[h], zn[h]), 0.f) * 0.999999f;
        const float tf = fminf(min3(xf[h], yf[h], zf[h]) * 1.000001f, c[h]);
        if (tn <= tf) key = min(key, __float_as_uint(tn));
    }
    return key;
}

// The closest hit in double (ties -> lowest face index) among a ray's first n
// candidates (32 entries apart) whose lower bound is within U; slot -1: none.
struct Hit { double t; int slot, id; };
__device__ __forceinline__ Hit closest_hit(const uint2* cand, int n, float U, const CTri* __restrict__ tris, float3 o,
                                           float3 d) {
    Hit h{1000.0, -1, -1};
    const d3 od = to_d3(o), dd = to_d3(d);
    for (int i = 0; i < n; ++i) {
        const uint2 e = cand[32 * i];
        if (__uint_as_float(e.y) > U) continue;
        const TriV t = load_tri(tris, (int)e.x);
        double t64;
        if (!ray_tri_d(od, dd, to_d3(t.a), to_d3(t.b), to_d3(t.c), 1000.0, &t64)) continue;
        if (t64 < h.t || (t64 == h.t && (h.slot < 0 || t.id < h.id))) h = Hit{t64, (int)e.x, t.id};
    }
    return h;
}
// A list that the walk has filled holds only its closest hit afterwards, whose
// distance bounds U.  Lists fill where more triangles than they hold may be
// the closest hit: faces that are there several times, or edge-on ones at a
// silhouette.  Settled where the walk meets them they cost their own double
// tests; a second walk of each such ray, by one lane, held whole launches (1M
// parallel rays along a height field of 80k faces, 294 of them with a full
// list: 773 against 430 us a call; 12 copies of 5,120 faces, 65k rays 390
// against 260).
__device__ __forceinline__ void keep_hit(const Hit& h, uint2* cand, int& nc, float& U) {
    nc = 0;
    if (h.slot < 0) return;
    cand[0] = make_uint2((uint32_t)h.slot, __float_as_uint(__double2float_rd(h.t)));
    U = fminf(U, __double2float_ru(h.t));
    nc = 1;
}
// A ray's result.
__device__ __forceinline__ void write_hit(const Hit& h, int64_t q, float3 o, float3 d, float* __restrict__ pos,
                                          int64_t* __restrict__ face_id, float* __restrict__ depth) {
    depth[q] = __double2float_rn(h.t);
    pos[3 * q] = __double2float_rn(dA((double)o.x, dM(h.t, (double)d.x)));
    pos[3 * q + 1] = __double2float_rn(dA((double)o.y, dM(h.t, (double)d.y)));
    pos[3 * q + 2] = __double2float_rn(dA((double)o.z, dM(h.t, (double)d.z)));
    face_id[q] = h.slot >= 0 ? (int64_t)h.id : (int64_t)-1;
}

// closest_hit and keep_hit out of line, so that the walks keep their registers
// (inline in k_ray's loop: 33.5M camera rays 3.41 against 3.08 ms).
struct Settled { int n; float U; };
__device__ __noinline__ Settled settle_full(uint2* cand, int n, const CTri* __restrict__ tris, float3 o, float3 d, float U) {
    Settled e{0, U};
    keep_hit(closest_hit(cand, n, U, tris, o, d), cand, e.n, e.U);
    return e;
}

constexpr int kRayBlocks = 8;   // blocks of k_ray per SM
// Closest hit of 32 rays per warp (a packet: the rays of 4 consecutive
// entries of `order`, units of 8 consecutive rays sorted so that nearby ones
// are side by side (k_ray_order, which lists the coherent packets for this
// kernel and the others for k_ray_lanes; packets holding a ray that is not
// finite or has no direction are added to its list here): warp-uniform walk of the
// union of the rays' paths.  At an inner node lane 8 g + j tests child j
// against unit g in interval arithmetic: what its two halves' origins and
// directions lie within against the box's planes (group_entry).  Eight
// neighbouring pixels sweep nearly what they hit, so this keeps few children
// that no ray needs, for about 100 instructions a node where a test per ray
// and child with eight warp minima took 350 (33.5M camera rays on 82k faces:
// 5.46 -> 3.14 ms a call; 32 warps per SM, 16 would be 20 % slower; at 64
// registers 204 bytes of spill stores and 260 of loads).  Children go onto the
// warp's stack farthest entry first.  Each lane keeps U, an upper bound of its
// closest hit (certain FP32 hits: t + error bound), and a short list of
// triangles that may still be closer (certain or undecided hits whose lower
// bound is within U); the list is settled in double at the end, or when one of
// the warp's is full: exact t of the closest hit, ties -> lowest face index.
__global__ void __launch_bounds__(kQBlock, kRayBlocks) k_ray(int64_t n, const uint32_t* __restrict__ order,
                                                 const float* __restrict__ ro,
                                                 const float* __restrict__ rd, float* __restrict__ pos,
                                                 int64_t* __restrict__ face_id, float* __restrict__ depth,
                                                 const DeviceTree tree, unsigned long long* __restrict__ ctr,
                                                 int64_t grab, const uint32_t* __restrict__ packets,
                                                 const unsigned long long* __restrict__ packets_n,
                                                 uint32_t* __restrict__ lanes,
                                                 unsigned long long* __restrict__ lanes_n) {
    const CTri* __restrict__ tris = tree.tris;
    const int lane = threadIdx.x & 31;
    __shared__ uint2 s_stack[kQBlock / 32][kStack];
    __shared__ uint2 s_cand[kQBlock / 32][kCand + 4][32];
    uint2* stk = s_stack[threadIdx.x >> 5];
    uint2* cand = &s_cand[threadIdx.x >> 5][0][lane];   // the lane's candidates, 32 entries apart: slot, lower bound
    PacketQueue pq(ctr, (int64_t)*packets_n, grab);
    for (int64_t at = pq.take(); at >= 0; at = pq.take()) {
        const int64_t pk = __ldg(packets + at);
        const int64_t q = packet_ray(pk, lane, n, order);
        const bool act = q < n;
        const float3 o = act ? load3(ro, q) : make_float3(0.f, 0.f, 0.f);
        const float3 d = act ? load3(rd, q) : make_float3(1.f, 1.f, 1.f);
        const float dinf = f3inf(d);
        const bool odd = !(f3inf(o) < CUDART_INF_F && dinf > 0.f && dinf < CUDART_INF_F);   // NaN: odd
        if (__any_sync(kFull, odd)) {
            if (lane == 0) lanes[atomicAdd(lanes_n, 1ull)] = (uint32_t)pk;
            continue;
        }
        float U = act ? 1000.0f : -1.f;             // MAX_DIST
        int nc = 0, sp = 0, cur = 0;
        bool live = true;
        while (true) {   // the walk, anew after the lists have been settled because one was full
            const RayAxis X = ray_axis(o.x, d.x, dinf, act), Y = ray_axis(o.y, d.y, dinf, act), Z = ray_axis(o.z, d.z, dinf, act);
            const bool mixed = __any_sync(kFull, X.kind == 2 || Y.kind == 2 || Z.kind == 2);
            float c[2];                                 // bounds of the lane's quad and of the other one
            uint32_t cullmax;
            auto share_bounds = [&]() {
                float m = act ? U * 1.000002f : -1.f;
                cullmax = __reduce_max_sync(kFull, __float_as_uint(fmaxf(m, 0.f)));
                m = fmaxf(m, __shfl_xor_sync(kFull, m, 1));
                c[0] = fmaxf(m, __shfl_xor_sync(kFull, m, 2));
                c[1] = __shfl_xor_sync(kFull, c[0], 4);
            };
            share_bounds();
            bool full = false;
            while (live && !full) {
                if (cur >= 0) {
                    const float4* nb = reinterpret_cast<const float4*>(tree.wnodes + cur);
                    const int j = lane & 7;
                    const float4 lo = __ldg(nb + j), hi = __ldg(nb + 8 + j);
                    uint32_t key = mixed ? group_entry<true>(X, Y, Z, lo, hi, c) : group_entry<false>(X, Y, Z, lo, hi, c);
                    key = min(key, __shfl_xor_sync(kFull, key, 8));
                    key = min(key, __shfl_xor_sync(kFull, key, 16));
                    if (key != kFull) key = (key & ~7u) | (uint32_t)j;
                    // its place on the stack: the number of needed children farther than it, two of
                    // the eight compared by each of the four lanes with this child
                    const uint32_t ka = __shfl_sync(kFull, key, 2 * (lane >> 3)), kb = __shfl_sync(kFull, key, 2 * (lane >> 3) + 1);
                    int place = (ka > key && ka != kFull ? 1 : 0) + (kb > key && kb != kFull ? 1 : 0);
                    place += __shfl_xor_sync(kFull, place, 8);
                    place += __shfl_xor_sync(kFull, place, 16);
                    const int kept = __popc(__ballot_sync(kFull, key != kFull) & 0xFFu);
                    __syncwarp();   // the popped entry has been read
                    if (lane < 8 && key != kFull) stk[sp + place] = make_uint2((uint32_t)__float_as_int(lo.w), key & ~7u);
                    sp += kept;
                    __syncwarp();
                } else {
                    int s0, s1;
                    leaf_range(cur, s0, s1);
                    const float U0 = U;
                    for (int s = s0; s < s1; ++s) {
                        const TriV t = load_tri(tris, s);
                        float tt, terr;
                        const int r = ray_tri_f(o, d, dinf, t, 1000.0f, &tt, &terr);
                        const float lb = tt - terr;
                        if (act && r != 0 && lb <= U) {
                            if (r == 1) U = fminf(U, tt + terr);
                            cand[32 * nc] = make_uint2((uint32_t)s, __float_as_uint(lb));
                            ++nc;
                        }
                    }
                    full = __any_sync(kFull, nc > kCand);
                    if (__any_sync(kFull, U < U0)) share_bounds();
                }
                // the next entry that some ray still needs
                live = false;
                while (sp > 0) {
                    const uint2 e = stk[--sp];
                    if (e.y <= cullmax) { cur = (int)e.x; live = true; break; }
                }
            }
            if (!live) break;
            const Settled e = settle_full(cand, nc, tris, o, d, U);
            nc = e.n;
            U = e.U;
        }
        if (act) write_hit(closest_hit(cand, nc, U, tris, o, d), q, o, d, pos, face_id, depth);
    }
}

// ------------------------------------------------------ Morton bucketing
// Points are counted into 2^(3b) cells of their own bounding box (computed
// on the device) and scattered in Morton order of the cells.  Within a cell
// the order is that of the atomics (irrelevant: results are per query).
__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // 10 bits -> every third bit
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
// order-preserving float <-> uint32 map (for atomicMin / atomicMax)
__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}
__global__ void k_box_init(uint32_t* box) {
    if (threadIdx.x < 3) box[threadIdx.x] = 0xFFFFFFFFu;
    else if (threadIdx.x < 6) box[threadIdx.x] = 0u;
}
__global__ void k_box(int64_t n, const float* __restrict__ pts, uint32_t* __restrict__ box) {
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0u, 0u, 0u};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float3 p = load3(pts, i);
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (isfinite(c[k])) { lo[k] = min(lo[k], f2o(c[k])); hi[k] = max(hi[k], f2o(c[k])); }
    }
    // one set of atomics a block: a set per warp, 57,000 atomics on six words,
    // took 41 us of 1M points' bucketing
    __shared__ uint32_t s_box[6];
    if (threadIdx.x < 6) s_box[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = __reduce_min_sync(kFull, lo[k]);
        hi[k] = __reduce_max_sync(kFull, hi[k]);
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) { atomicMin(&s_box[k], lo[k]); atomicMax(&s_box[3 + k], hi[k]); }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&box[threadIdx.x], s_box[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&box[threadIdx.x], s_box[threadIdx.x]);
}
__device__ __forceinline__ uint32_t cell_of(float3 p, const uint32_t* __restrict__ box, int bits) {
    const float side = (float)(1 << bits), m = side - 1.f;
    const float c[3] = {p.x, p.y, p.z};
    uint32_t g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = o2f(box[k]), hi = o2f(box[3 + k]);
        const float s = hi > lo ? side / (hi - lo) : 0.f;
        const float v = (c[k] - lo) * s;
        g[k] = (uint32_t)fminf(fmaxf(v == v ? v : 0.f, 0.f), m);
    }
    return spread3(g[0]) | (spread3(g[1]) << 1) | (spread3(g[2]) << 2);
}
__global__ void k_cell_hist(int64_t n, const float* __restrict__ pts, const uint32_t* __restrict__ box, int bits,
                            uint32_t* __restrict__ hist) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        atomicAdd(&hist[cell_of(load3(pts, i), box, bits)], 1u);
}
__global__ void k_cell_scatter(int64_t n, const float* __restrict__ pts, const uint32_t* __restrict__ box, int bits,
                               uint32_t* __restrict__ offs, uint32_t* __restrict__ order) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        order[atomicAdd(&offs[cell_of(load3(pts, i), box, bits)], 1u)] = (uint32_t)i;
}

constexpr int kLaneBlocks = 6;    // blocks of k_ray_lanes per SM
constexpr int kLaneRefill = 16;   // idle lanes that make a warp finish them and take new rays
constexpr int kLaneInner = 12;    // fewer lanes at inner nodes than this wait for those at leaves
// the same for few rays, bound by the latency of a walk: registers without
// spills, and lanes at leaves wait less (1,000 rays on 1.3M faces 233 against
// 264 us; 5M rays 2.31 against 2.08 ms)
constexpr int kFewLaneBlocks = 4, kFewLaneInner = 4;
// Closest hit of the rays of the incoherent packets (k_ray_order and k_ray
// list them): each lane walks its own ray alone (own stack in local memory,
// children nearest first, a child popped only while its entry distance is
// within the lane's bound U).  The warp keeps its lanes on the same kind of
// step, inner nodes until few lanes are at one, then leaves; rays that ended
// wait until kLaneRefill lanes are idle, which settle their hits in double
// together and take the next rays of the warp's packet.  A warp that walked
// its 32 rays to the longest one's end had 6.8 lanes active and took 497
// instructions a ray; refilled, with two children an instruction in
// affine_pair, 11.3 and 287: 5M random rays on 82k faces 3.36 -> 2.32 ms a call
// (refill at 8 or 4 idle lanes 3 and 9 % slower, leaves at once 13 %), 2.08 with
// full lists settled out of line; what is left is load latency and divergence
// (80 registers, 94 bytes of spill stores and 104 of loads).  Filters, candidate
// list and the FP64 settlement are k_ray's, so every result is the one k_ray
// would give.
template <bool FEW>
__global__ void __launch_bounds__(kQBlock, FEW ? kFewLaneBlocks : kLaneBlocks) k_ray_lanes(int64_t n, const uint32_t* __restrict__ order,
                                                       const float* __restrict__ ro, const float* __restrict__ rd,
                                                       float* __restrict__ pos, int64_t* __restrict__ face_id,
                                                       float* __restrict__ depth, const CNode* __restrict__ nodes,
                                                       const CTri* __restrict__ tris,
                                                       const uint32_t* __restrict__ lanes,
                                                       const unsigned long long* __restrict__ lanes_n,
                                                       unsigned long long* __restrict__ next) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ uint2 s_cand[kQBlock / 32][kCand][32];
    uint2* cand = &s_cand[threadIdx.x >> 5][0][lane];   // the lane's candidates, 32 entries apart: slot, lower bound
    const unsigned long long count = *lanes_n;
    uint2 st[kStack];
    int sp = 0, cur = 0, nc = 0;
    bool live = false;                       // the lane's walk goes on
    int64_t q = -1;                          // the lane's ray, -1: none
    float3 o = make_float3(0.f, 0.f, 0.f), d = o, inv = o;
    float dinf = 0.f, U = 0.f;
    bool degen = false;
    int64_t packet = -1;                     // the warp's packet, its next ray (32: used up), more may come
    int from = 32;
    bool more = true;
    while (true) {
        const unsigned idle = __ballot_sync(kFull, !live);
        if (idle == kFull || (more && __popc(idle) >= kLaneRefill)) {
            if (!live && q >= 0) {           // settle and write
                write_hit(closest_hit(cand, nc, U, tris, o, d), q, o, d, pos, face_id, depth);
                q = -1;
            }
            __syncwarp();
            if (from >= 32 && more) {        // the warp's next packet
                unsigned long long c = 0;
                if (lane == 0) c = atomicAdd(next, 1ull);
                c = __shfl_sync(kFull, c, 0);
                more = c < count;
                if (more) { packet = (int64_t)__ldg(lanes + c); from = 0; }
            }
            if (from < 32) {
                const int k = from + __popc(idle & lt);
                if (!live && k < 32) {
                    q = packet_ray(packet, k, n, order);
                    if (q >= n) q = -1;
                    if (q >= 0) {
                        o = load3(ro, q);
                        d = load3(rd, q);
                        inv = ray_inv(d);
                        degen = ray_degenerate(inv);
                        dinf = f3inf(d);
                        U = 1000.0f;         // MAX_DIST
                        nc = sp = cur = 0;
                        live = true;
                    }
                }
                from = min(32, from + __popc(idle));
            } else if (idle == kFull) {
                break;                       // no ray left
            }
            continue;
        }
        // inner nodes
        while (true) {
            const unsigned in = __ballot_sync(kFull, live && cur >= 0);
            if (!in || (__popc(in) < (FEW ? kFewLaneInner : kLaneInner) && __any_sync(kFull, live && cur < 0))) break;
            if (live && cur >= 0) {
                const float cull = U * 1.000002f;
                const NodeView nd = load_node(nodes, cur);
                uint32_t k[8];
                lane_child_keys(nd, o, inv, degen, cull, k);
                sort8(k);
#pragma unroll
                for (int i = 7; i >= 1; --i)
                    if (k[i] != kFull) st[sp++] = make_uint2((uint32_t)child_ref(nd, meta_of(nd, (int)(k[i] & 7u))), k[i] & ~7u);
                if (k[0] != kFull) {
                    cur = child_ref(nd, meta_of(nd, (int)(k[0] & 7u)));
                } else {                     // the next entry whose box is still within the bound
                    live = false;
                    while (sp > 0) {
                        const uint2 e = st[--sp];
                        if (__uint_as_float(e.y) <= cull) { cur = (int)e.x; live = true; break; }
                    }
                }
            }
            if (more && __popc(__ballot_sync(kFull, !live)) >= kLaneRefill) break;
        }
        // leaves
        if (live && cur < 0) {
            int s0, s1;
            leaf_range(cur, s0, s1);
            for (int s = s0; s < s1; ++s) {
                const TriV t = load_tri(tris, s);
                float tt, terr;
                const int r = ray_tri_f(o, d, dinf, t, 1000.0f, &tt, &terr);
                const float lb = tt - terr;
                if (r != 0 && lb <= U) {
                    if (r == 1) U = fminf(U, tt + terr);
                    if (nc == kCand) {   // keep only live candidates
                        nc = 0;
                        for (int i = 0; i < kCand; ++i)
                            if (__uint_as_float(cand[32 * i].y) <= U) { cand[32 * nc] = cand[32 * i]; ++nc; }
                        if (nc == kCand) {
                            const Settled e = settle_full(cand, kCand, tris, o, d, U);
                            nc = e.n;
                            U = e.U;
                        }
                    }
                    cand[32 * nc] = make_uint2((uint32_t)s, __float_as_uint(lb));
                    ++nc;
                }
            }
            const float cull = U * 1.000002f;
            live = false;
            while (sp > 0) {
                const uint2 e = st[--sp];
                if (__uint_as_float(e.y) <= cull) { cur = (int)e.x; live = true; break; }
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------- ray windows
// Packet order of rays.  Rays are taken in units of kUnit consecutive rays,
// and each window of kOrdUnits consecutive units is sorted by the Morton
// code of the point where one ray of the unit (its fourth) enters the root
// node's box (its origin when it starts inside), on cells of one size on all
// three axes (the window's largest extent / 1024); units whose ray misses
// the box go after the others, in the Morton order of where that ray passes
// closest to the box centre (clamped into the cells), then the window's tail
// past the last unit.  A packet is four consecutive units of the sorted
// order.  Camera rays stored row by row then make packets of 8 pixels from
// each of 4 neighbouring rows instead of 32 x 1 strips, and the union of the
// 32 rays' walks visits far fewer nodes (33.5M camera rays: k_ray 6.4 -> 5.1
// ms when it tested every ray, for a sort of 1,024 keys per 8,192 rays, 0.22
// ms).  The order changes no result: each ray's hit is its own.
constexpr int kOrdThreads = 256, kOrdItems = 4;
constexpr int kOrdUnits = kOrdThreads * kOrdItems;    // 1024 units = 8192 rays per window
// Entry point of ray (o, d) into the box [lo, lo + 255 * 2^ex] (the origin when
// the ray starts inside; non-finite coordinates become 0): 0, or 1 when the
// ray misses the box (e = the point where it passes closest to the box
// centre, for t >= 0).
__device__ __forceinline__ int ray_entry(float3 o, float3 d, const float lo[3], const int ex[3], float e[3]) {
    const float oc[3] = {o.x, o.y, o.z}, dc[3] = {d.x, d.y, d.z};
    float tn = 0.f, tf = CUDART_INF_F;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float hi = fmaf(255.f, exp2i(ex[k]), lo[k]);
        const float inv = 1.f / dc[k];
        const float ta = (lo[k] - oc[k]) * inv, tb = (hi - oc[k]) * inv;
        tn = fmaxf(tn, fminf(ta, tb));   // NaN (0 * inf) leaves the bound as it was
        tf = fminf(tf, fmaxf(ta, tb));
    }
    const int miss = tn <= tf ? 0 : 1;
    if (miss) {                       // where the ray passes closest to the box centre
        float cd = 0.f, dd = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float c = 0.5f * (lo[k] + fmaf(255.f, exp2i(ex[k]), lo[k]));
            cd = fmaf(c - oc[k], dc[k], cd);
            dd = fmaf(dc[k], dc[k], dd);
        }
        tn = fmaxf(cd / dd, 0.f);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float v = fmaf(dc[k], tn, oc[k]);
        e[k] = isfinite(v) ? v : 0.f;
    }
    return miss;
}
// One block per window: entry points of the units' rays, the box of those
// that enter, Morton keys, a block radix sort of (key, unit in the window),
// and the sorted unit indices written to order[].  Then each packet of the
// window (4 consecutive sorted units) is judged by the first and last rays of
// its units against their fourth, and by the fourths (above); face: the
// density of the mesh, 1 / sqrt(faces).  The packets to trace as such are
// listed for k_ray, the others for k_ray_lanes (with a flag per packet instead,
// k_ray took 359 us to pass over the packets of 16.8M incoherent rays: an
// atomic each on its queue; 5M such rays 2.31 -> 2.20 ms a call).
__global__ void __launch_bounds__(kOrdThreads) k_ray_order(int64_t n, const float* __restrict__ ro,
                                                           const float* __restrict__ rd,
                                                           const CNode* __restrict__ nodes, float face,
                                                           uint32_t* __restrict__ order, uint32_t* __restrict__ packets,
                                                           unsigned long long* __restrict__ packets_n,
                                                           uint32_t* __restrict__ lanes,
                                                           unsigned long long* __restrict__ lanes_n) {
    using Sort = cub::BlockRadixSort<uint32_t, kOrdThreads, kOrdItems, uint16_t>;
    __shared__ typename Sort::TempStorage s_sort;
    __shared__ uint32_t s_box[6];
    __shared__ float s_ray[kOrdUnits][6];     // each unit's fourth ray: unit direction, origin
    __shared__ uint8_t s_bad[kOrdUnits];       // the unit's first or last ray strays from its fourth: beyond the limits 1, twice 2
    __shared__ uint16_t s_sorted[kOrdUnits];
    const int64_t units = (n + kUnit - 1) / kUnit;
    const int64_t u0 = (int64_t)blockIdx.x * kOrdUnits;
    const int t = threadIdx.x;
    if (t < 3) s_box[t] = 0xFFFFFFFFu;
    else if (t < 6) s_box[t] = 0u;
    const NodeView root = load_node(nodes, 0);
    const float blo[3] = {root.ox, root.oy, root.oz};
    const int bex[3] = {nodes[0].ex, nodes[0].ey, nodes[0].ez};
    const float strict = n < kFewRays ? kCohFew : 1.f;
    const float extent = 255.f * fmaxf(fmaxf(root.sx, root.sy), root.sz);
    const float spread_max = strict * kCohOrigin * extent;
    float ep[kOrdItems][3];
    int kind[kOrdItems];              // 0 enters the box, 1 misses it, 2 past the last unit
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < kOrdItems; ++i) {
        const int li = i * kOrdThreads + t;
        const int64_t u = u0 + li;
        kind[i] = 2;
        ep[i][0] = ep[i][1] = ep[i][2] = 0.f;
        if (u >= units) continue;
        const int64_t q = min(u * kUnit + kUnit / 2 - 1, n - 1);
        const float3 o = load3(ro, q), d = load3(rd, q);
        kind[i] = ray_entry(o, d, blo, bex, ep[i]);
        if (kind[i] == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) { lo[k] = min(lo[k], f2o(ep[i][k])); hi[k] = max(hi[k], f2o(ep[i][k])); }
        }
        const float il = rsqrtf(f3dot(d, d));
        const float3 v = make_float3(d.x * il, d.y * il, d.z * il);
        const float3 far = f3sub(make_float3(ep[i][0], ep[i][1], ep[i][2]), o);
        const float dir_max = strict * fminf(kCohDir, kCohFaces * face * extent * rsqrtf(f3dot(far, far)));
        // a finite fourth direction, not zero (NaN: bad); within the limits, within twice the limits
        bool in = f3inf(v) <= 2.f, near = in;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t qe = e == 0 ? u * kUnit : min(u * kUnit + kUnit - 1, n - 1);
            const float3 oe = load3(ro, qe), de = load3(rd, qe);
            const float ie = rsqrtf(f3dot(de, de));
            const float dv = f3inf(f3sub(make_float3(de.x * ie, de.y * ie, de.z * ie), v)), dov = f3inf(f3sub(oe, o));
            in &= dv <= dir_max && dov <= spread_max;
            near &= dv <= 2.f * dir_max && dov <= 2.f * spread_max;
        }
        s_ray[li][0] = v.x; s_ray[li][1] = v.y; s_ray[li][2] = v.z;
        s_ray[li][3] = o.x; s_ray[li][4] = o.y; s_ray[li][5] = o.z;
        s_bad[li] = in ? 0 : (near ? 1 : 2);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = __reduce_min_sync(kFull, lo[k]);
        hi[k] = __reduce_max_sync(kFull, hi[k]);
    }
    __syncthreads();                  // s_box initialised
    if ((t & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) { atomicMin(&s_box[k], lo[k]); atomicMax(&s_box[3 + k], hi[k]); }
    }
    __syncthreads();
    float wlo[3], ext = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        wlo[k] = o2f(s_box[k]);
        ext = fmaxf(ext, o2f(s_box[3 + k]) - wlo[k]);   // no entry point: the box is empty, ext stays 0
    }
    const float sc = ext > 0.f ? 1024.f / ext : 0.f;
    uint32_t key[kOrdItems];
    uint16_t val[kOrdItems];
#pragma unroll
    for (int i = 0; i < kOrdItems; ++i) {
        val[i] = (uint16_t)(i * kOrdThreads + t);
        if (kind[i] == 2) { key[i] = 0x80000000u; continue; }
        uint32_t g[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) g[k] = (uint32_t)fminf(fmaxf((ep[i][k] - wlo[k]) * sc, 0.f), 1023.f);
        key[i] = spread3(g[0]) | (spread3(g[1]) << 1) | (spread3(g[2]) << 2) | (kind[i] == 1 ? 0x40000000u : 0u);
    }
    Sort(s_sort).SortBlockedToStriped(key, val, 0, 32);
#pragma unroll
    for (int i = 0; i < kOrdItems; ++i) {
        const int rank = i * kOrdThreads + t;            // rank of the window
        s_sorted[rank] = val[i];
        if (u0 + rank < units) order[u0 + rank] = (uint32_t)(u0 + val[i]);
    }
    __syncthreads();
    // packet t of the window: sorted units 4t .. 4t + 3
    const int64_t pk = (int64_t)blockIdx.x * (kOrdUnits / 4) + t;
    const bool valid = u0 + 4 * t < units;
    int bad = 0;
    if (valid) {
        const int f = s_sorted[4 * t];
        bad = s_bad[f];
        for (int j = 1; j < 4 && u0 + 4 * t + j < units; ++j) {
            const int v = s_sorted[4 * t + j];
            float dv = 0.f, dov = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                dv = fmaxf(dv, fabsf(s_ray[v][k] - s_ray[f][k]));
                dov = fmaxf(dov, fabsf(s_ray[v][3 + k] - s_ray[f][3 + k]));
            }
            const bool in = dv <= kCohUnits && dov <= spread_max, near = dv <= 2.f * kCohUnits && dov <= 2.f * spread_max;
            bad = max(bad, max((int)s_bad[v], in ? 0 : (near ? 1 : 2)));
        }
    }
    // the window's packets go one way, but for those beyond twice the limits
    const int total = __syncthreads_count(valid), in_limits = __syncthreads_count(valid && bad == 0);
    const bool inc = 2 * in_limits < total || bad == 2;
    auto list = [&](bool in, uint32_t* __restrict__ to, unsigned long long* __restrict__ to_n) {
        const unsigned m = __ballot_sync(kFull, in);
        if (m) {                      // one atomic per warp
            unsigned long long base = 0;
            if ((t & 31) == __ffs(m) - 1) base = atomicAdd(to_n, (unsigned long long)__popc(m));
            base = __shfl_sync(kFull, base, __ffs(m) - 1);
            if (in) to[base + __popc(m & ((1u << (t & 31)) - 1u))] = (uint32_t)pk;
        }
    };
    list(valid && !inc, packets, packets_n);
    list(valid && inc, lanes, lanes_n);
}

// --------------------------------------------------------------- launchers
namespace {

int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}
template <class K>
unsigned persistent_grid(K kernel, int64_t n) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kQBlock, 0);
    if (per_sm < 1) per_sm = 1;
    const int64_t want = (n + kQBlock - 1) / kQBlock;
    const int64_t cap = (int64_t)sm_count() * per_sm;
    return (unsigned)(want < cap ? (want > 0 ? want : 1) : cap);
}

int cell_bits(int64_t n) {
    int b = 4;
    while (b < 8 && ((int64_t)1 << (3 * (b + 1))) <= 2 * n) ++b;
    return b;
}

}  // namespace

// Heavy-query list length for n queries: a 32nd of them, at least 262,144
// (4 MB), at most n: a launch of few packets per warp may hand most of its
// queries over.  A full list only means packets finish in place.
int64_t heavy_cap_for(int64_t n) {
    const int64_t c = n / 32 > (1 << 18) ? n / 32 : (1 << 18);
    return c < n ? c : n;
}

namespace {
// Ray launch workspace: counters (256 bytes), the unit order, the lists of
// coherent and of incoherent packets; byte offsets and total.
struct RayWs { size_t order, packets, lanes, end; };
RayWs ray_ws(int64_t n) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t units = (size_t)((n + kUnit - 1) / kUnit), packets = (size_t)((n + 31) / 32);
    RayWs r;
    r.order = 256;
    r.packets = r.order + al(sizeof(uint32_t) * units);
    r.lanes = r.packets + al(sizeof(uint32_t) * packets);
    r.end = r.lanes + al(sizeof(uint32_t) * packets);
    return r;
}
}  // namespace

size_t query_workspace_bytes(int mode, int64_t n) {
    size_t b = 256;                                               // packet counters
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    if (mode >= 0 && n >= kFewQueries) {
        const int64_t cells = (int64_t)1 << (3 * cell_bits(n));
        b += al(sizeof(uint32_t) * n);                            // order
        b += al(sizeof(uint32_t) * (cells + 1));                  // cell counts / offsets
        b += al(sizeof(uint32_t) * (scan::num_chunks(cells) + 1));
        b += al(sizeof(uint32_t) * 8);                            // query box
    }
    if (mode > 0) b += al(sizeof(int32_t) * n);                   // winning slots
    if (mode == 1) b += al(sizeof(uint32_t) * n);                 // watertight overflow queue
    if (mode >= 0) b += al(sizeof(uint4) * heavy_cap_for(n));     // heavy-query list
    if (mode == 2) b += al(sizeof(uint4) * n);                    // raystab candidates (second pass)
    if (mode == -1) b = ray_ws(n).end;                           // unit order, coherent and incoherent packets
    return b;
}

namespace {
// Slots of the 256-byte counter block at the head of a launch's workspace
// (32 uint64, zeroed at the start of every launch); each has one user.
enum : int {
    kCtUdf = 0,         // k_udf packet queue
    kCtSign = 1,        // sign-pass packet queue (watertight, or the first raystab pass of a single BVH)
    kCtArenaRs = 2,     // first raystab pass of an arena (its watertight pass takes kCtSign)
    kCtHeavyN = 6,      // heavy-query list length
    kCtHeavyNext = 7,   // k_udf_heavy queue
    kCtOvfN = 10,       // watertight overflow queue length
    kCtCandN = 12,      // raystab second-pass candidates
    kCtLinesNext = 13,  // raystab second-pass queue
    kCtParity = 11,     // edge parity of a single BVH (k_edge_parity)
    kCtRayLanesN = 14,  // incoherent ray packets
    kCtRayLanesNext = 15,  // k_ray_lanes queue
    kCtLate = 8,        // k_udf packets in a long walk after the queue is empty
    kCtRayPacketsN = 16,   // coherent ray packets
};
// packets per atomic grab: about 64 grabs per warp
int64_t grab_for(int64_t n, unsigned grid) {
    const int64_t packets = (n + 31) / 32;
    const int64_t warps = (int64_t)grid * (kQBlock / 32);
    const int64_t g = packets / (warps * 64);
    return g < 1 ? 1 : g;
}
// Queue shape of k_udf: three quarters of the packets in runs of up to kRun
// neighbouring ones, the others as grab_for (k_udf's seeds; 16 and 8 measured slower on uneven
// work), at least about eight tickets per warp.
constexpr int64_t kRun = 4;
RunShape run_shape(int64_t n, unsigned grid) {
    const int64_t packets = (n + 31) / 32;
    const int64_t warps = (int64_t)grid * (kQBlock / 32);
    RunShape q{0, 1, grab_for(n, grid)};
    q.big = packets / (warps * 8);
    if (q.big > kRun) q.big = kRun;
    if (q.big <= q.grab) { q.big = 1; return q; }
    q.nbig = packets * 3 / 4 / q.big;
    return q;
}
// grabs that hand out the packets of n queries
int64_t grabs_for(int64_t n, unsigned grid) {
    const int64_t g = grab_for(n, grid);
    return ((n + 31) / 32 + g - 1) / g;
}
// Launch shape of a yielding launch (PacketQueue block budget): kYieldWaves
// times the persistent grid g, each block taking at most block_grabs grabs,
// twice the queue's grabs in all, so the queue is always drained (a warp
// stops only when its block's budget is spent or the queue is empty) and a
// block lives for about 1 / (kYieldWaves / 2) of the launch.  off: the
// persistent launch (g blocks, no budget).
constexpr unsigned kYieldWaves = 4;  // measured against 8 and 16
struct LaunchShape { unsigned grid; int block_grabs; };
LaunchShape yield_shape(unsigned g, int64_t grabs, bool on) {
    if (!on) return {g, 0};
    int64_t G = (int64_t)g * kYieldWaves;
    if (G > 2 * grabs) G = 2 * grabs > 0 ? 2 * grabs : 1;
    const int64_t bg = (2 * grabs + G - 1) / G;
    return {(unsigned)G, (int)(bg > 0 ? bg : 1)};
}
// raystab chunk: kChunkMax packets, one packet when the launch has few per warp
int64_t chunk_for(int64_t n, unsigned grid) {
    const int64_t packets = (n + 31) / 32;
    const int64_t warps = (int64_t)grid * (kQBlock / 32);
    return packets >= (int64_t)kChunkMax * warps ? kChunkMax : 1;
}
}  // namespace

namespace {
// Rays the first raystab pass traces per query before handing the query to
// the second pass (a line of two rays per stab direction).
constexpr int kRaystabFirstRays = 2;
// The two raystab passes over the packets of `w` (n queries): counters ctr
// (first pass), cand_n (candidates appended), lines_next (second-pass
// queue) and the edge parities (k_edge_parity), all zero; cand holds up to n candidates.
void launch_raystab(const Work& w, int64_t n, const uint32_t* order, const float* pts, float* dist,
                    const CNode* nodes, const CTri* tris, unsigned long long* ctr, uint4* cand,
                    unsigned long long* cand_n, unsigned long long* lines_next, int64_t n_tris,
                    const int64_t* face_off, const int32_t* face_slot, int n_meshes, unsigned long long* parity,
                    cudaStream_t stream) {
    k_edge_parity<<<(unsigned)((n_tris + 1023) / 1024), 256, 0, stream>>>(n_tris, tris, face_off, face_slot, n_meshes,
                                                                          parity); count_launch();
    const unsigned g = persistent_grid(k_sign_raystab, n);
    k_sign_raystab<<<g, kQBlock, 0, stream>>>(w, order, pts, dist, nodes, tris, ctr, chunk_for(n, g), cand, cand_n, parity);
    count_launch();
    const unsigned g2 = persistent_grid(k_sign_raystab_lines, n);
    k_sign_raystab_lines<<<g2, kQBlock, 0, stream>>>(pts, dist, nodes, tris, cand, cand_n, lines_next,
                                                     kRaystabFirstRays); count_launch();
}
}  // namespace

namespace {
template <bool UVW, bool SLOT>
void launch_few_t(int64_t n, const float* pts, float* dist, int64_t* fid, float* uvw, int32_t* slots,
                  const DeviceTree& tree, const MeshDesc* meshes, const int64_t* qoff, int n_meshes, int slot0,
                  cudaStream_t stream) {
    const int64_t room = (int64_t)sm_count() * kFewWarps;
    const int q = n <= room ? 1 : (n <= 2 * room ? 2 : 4);   // queries per warp
    const int64_t warps = (n + q - 1) / q;
    k_udf_few<UVW, SLOT><<<(unsigned)((warps + 3) / 4), kQBlock, 0, stream>>>(n, pts, dist, fid, uvw, slots, tree, meshes,
                                                                              qoff, n_meshes, slot0, q); count_launch();
}
void launch_few(int64_t n, const float* pts, float* dist, int64_t* fid, float* uvw, int32_t* slots,
                const DeviceTree& tree, const MeshDesc* meshes, const int64_t* qoff, int n_meshes, int slot0,
                cudaStream_t stream) {
    if (uvw && slots) launch_few_t<true, true>(n, pts, dist, fid, uvw, slots, tree, meshes, qoff, n_meshes, slot0, stream);
    else if (uvw) launch_few_t<true, false>(n, pts, dist, fid, uvw, slots, tree, meshes, qoff, n_meshes, slot0, stream);
    else if (slots) launch_few_t<false, true>(n, pts, dist, fid, uvw, slots, tree, meshes, qoff, n_meshes, slot0, stream);
    else launch_few_t<false, false>(n, pts, dist, fid, uvw, slots, tree, meshes, qoff, n_meshes, slot0, stream);
}
template <bool UVW, bool SLOT>
void launch_nearest_t(const Work& w, int64_t n, const uint32_t* order, const float* pts, float* dist, int64_t* fid,
                      float* uvw, int32_t* slots, const DeviceTree& tree, uint4* heavy, int64_t hcap,
                      unsigned long long* ctr, bool yield, cudaStream_t stream) {
    const unsigned g = persistent_grid(k_udf<UVW, SLOT>, n);
    const RunShape q = run_shape(n, g);
    const LaunchShape y = yield_shape(g, q.tickets(w.packets()), yield);
    k_udf<UVW, SLOT><<<y.grid, kQBlock, 0, stream>>>(w, order, pts, dist, fid, uvw, slots, tree, ctr + kCtUdf, q, heavy,
                                                     ctr + kCtHeavyN, hcap, ctr + kCtLate, y.block_grabs); count_launch();
    const unsigned gh = persistent_grid(k_udf_heavy<UVW, SLOT>, 32 * hcap);
    k_udf_heavy<UVW, SLOT><<<gh, kQBlock, 0, stream>>>(heavy, ctr + kCtHeavyN, hcap, w.meshes, w.slot0, pts, dist, fid, uvw,
                                                       slots, tree, ctr + kCtHeavyNext); count_launch();
}
// The distance search over the packets of `w` (n queries): the packets, then
// the queries they left to k_udf_heavy.
void launch_nearest(const Work& w, int64_t n, const uint32_t* order, const float* pts, float* dist, int64_t* fid,
                    float* uvw, int32_t* slots, const DeviceTree& tree, uint4* heavy, int64_t hcap,
                    unsigned long long* ctr, bool yield, cudaStream_t stream) {
    if (uvw && slots) launch_nearest_t<true, true>(w, n, order, pts, dist, fid, uvw, slots, tree, heavy, hcap, ctr, yield, stream);
    else if (uvw) launch_nearest_t<true, false>(w, n, order, pts, dist, fid, uvw, slots, tree, heavy, hcap, ctr, yield, stream);
    else if (slots) launch_nearest_t<false, true>(w, n, order, pts, dist, fid, uvw, slots, tree, heavy, hcap, ctr, yield, stream);
    else launch_nearest_t<false, false>(w, n, order, pts, dist, fid, uvw, slots, tree, heavy, hcap, ctr, yield, stream);
}
}  // namespace

cudaError_t launch_distance(int mode, bool want_uvw, int64_t n, const float* pts, float* dist, int64_t* fid,
                            float* uvw, const DeviceTree& tree, int slot_face0, NearLists near,
                            void* ws, cudaStream_t stream, int64_t qbase, bool yield) {
    if (n <= 0) return cudaSuccess;
    const CNode* nodes = tree.nodes;
    const CTri* tris = tree.tris;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    char* w = static_cast<char*>(ws);
    unsigned long long* ctr = reinterpret_cast<unsigned long long*>(w); w += 256;
    const bool few = n < kFewQueries;
    cudaError_t e = cudaSuccess;
    if (!(few && mode == 0) && (e = cudaMemsetAsync(ctr, 0, 256, stream)) != cudaSuccess) return e;
    uint32_t* order = nullptr;
    if (!few) {
        const int bits = cell_bits(n);
        const int64_t cells = (int64_t)1 << (3 * bits);
        order = reinterpret_cast<uint32_t*>(w); w += al(sizeof(uint32_t) * n);
        uint32_t* hist = reinterpret_cast<uint32_t*>(w); w += al(sizeof(uint32_t) * (cells + 1));
        uint32_t* bsum = reinterpret_cast<uint32_t*>(w); w += al(sizeof(uint32_t) * (scan::num_chunks(cells) + 1));
        uint32_t* box = reinterpret_cast<uint32_t*>(w); w += al(sizeof(uint32_t) * 8);
        if ((e = cudaMemsetAsync(hist, 0, sizeof(uint32_t) * (cells + 1), stream)) != cudaSuccess) return e;
        const unsigned g = (unsigned)sm_count() * 8;
        k_box_init<<<1, 32, 0, stream>>>(box); count_launch();
        k_box<<<g, 256, 0, stream>>>(n, pts, box); count_launch();
        k_cell_hist<<<g, 256, 0, stream>>>(n, pts, box, bits, hist); count_launch();
        scan::exclusive(hist, bsum, cells, stream);
        k_cell_scatter<<<g, 256, 0, stream>>>(n, pts, box, bits, hist, order); count_launch();
    }
    int32_t* slots = mode != 0 ? reinterpret_cast<int32_t*>(w) : nullptr;
    if (mode != 0) w += al(sizeof(int32_t) * n);
    uint32_t* ovf = mode == 1 ? reinterpret_cast<uint32_t*>(w) : nullptr;
    if (mode == 1) w += al(sizeof(uint32_t) * n);
    uint4* heavy = reinterpret_cast<uint4*>(w);
    const int64_t hcap = heavy_cap_for(n);
    w += al(sizeof(uint4) * hcap);
    const Work work{nullptr, nullptr, n, slot_face0, qbase};
    if (few)
        launch_few(n, pts, dist, fid, want_uvw ? uvw : nullptr, slots, tree, nullptr, nullptr, 0, slot_face0, stream);
    else
        launch_nearest(work, n, order, pts, dist, fid, want_uvw ? uvw : nullptr, slots, tree, heavy, hcap, ctr, yield, stream);
    if (mode == 1) {
        if (near.cnt) {
            const unsigned g = persistent_grid(k_sign_watertight<true>, n);
            const LaunchShape y = yield_shape(g, grabs_for(n, g), yield);
            k_sign_watertight<true><<<y.grid, kQBlock, 0, stream>>>(work, order, pts, dist, slots, nodes, tris, tree.wtris, near, ovf,
                                                                    ctr + kCtOvfN, ctr + kCtSign, grab_for(n, g),
                                                                    y.block_grabs); count_launch();
            if (near.ovf) {
                const unsigned go = persistent_grid(k_sign_watertight_ovf, n);
                k_sign_watertight_ovf<<<go, kQBlock, 0, stream>>>(ovf, ctr + kCtOvfN, pts, dist, slots, nodes, tris); count_launch();
            }
        } else {
            const unsigned g = persistent_grid(k_sign_watertight<false>, n);
            const LaunchShape y = yield_shape(g, grabs_for(n, g), yield);
            k_sign_watertight<false><<<y.grid, kQBlock, 0, stream>>>(work, order, pts, dist, slots, nodes, tris, tree.wtris, near,
                                                                     nullptr, nullptr, ctr + kCtSign, grab_for(n, g),
                                                                     y.block_grabs); count_launch();
        }
    } else if (mode == 2) {
        uint4* cand = reinterpret_cast<uint4*>(w);
        launch_raystab(work, n, order, pts, dist, nodes, tris, ctr + kCtSign, cand, ctr + kCtCandN, ctr + kCtLinesNext,
                       tree.n_tris, nullptr, nullptr, 1, ctr + kCtParity, stream);
    }
    return cudaGetLastError();
}

cudaError_t launch_near_lists(int64_t n_tris, const CNode* nodes, const CTri* tris, int32_t* cnt, int32_t* lst,
                              double* nrm, int* any_ovf, cudaStream_t stream) {
    if (n_tris <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(any_ovf, 0, sizeof(int), stream);
    if (e != cudaSuccess) return e;
    const unsigned g = persistent_grid(k_near_lists, n_tris);
    k_near_lists<<<g, kQBlock, 0, stream>>>(n_tris, nodes, tris, 0, cnt, lst, nrm, any_ovf); count_launch();
    return cudaGetLastError();
}

cudaError_t launch_ray(int64_t n, const float* ro, const float* rd, float* pos, int64_t* fid, float* depth,
                       const DeviceTree& tree, void* ws, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const CNode* nodes = tree.nodes;
    const CTri* tris = tree.tris;
    unsigned long long* ctr = reinterpret_cast<unsigned long long*>(ws);
    cudaError_t e = cudaMemsetAsync(ctr, 0, 256, stream);
    if (e != cudaSuccess) return e;
    const RayWs r = ray_ws(n);
    char* w = static_cast<char*>(ws);
    uint32_t* order = reinterpret_cast<uint32_t*>(w + r.order);
    uint32_t* packets = reinterpret_cast<uint32_t*>(w + r.packets);
    uint32_t* lanes = reinterpret_cast<uint32_t*>(w + r.lanes);
    const int64_t units = (n + kUnit - 1) / kUnit;
    k_ray_order<<<(unsigned)((units + kOrdUnits - 1) / kOrdUnits), kOrdThreads, 0, stream>>>(
        n, ro, rd, nodes, 1.f / sqrtf((float)tree.n_tris), order, packets, ctr + kCtRayPacketsN, lanes, ctr + kCtRayLanesN);
    count_launch();
    const unsigned g = persistent_grid(k_ray, n);
    k_ray<<<g, kQBlock, 0, stream>>>(n, order, ro, rd, pos, fid, depth, tree, ctr + kCtUdf, grab_for(n, g), packets,
                                     ctr + kCtRayPacketsN, lanes, ctr + kCtRayLanesN); count_launch();
    if (n < kFewRays) {
        const unsigned gl = persistent_grid(k_ray_lanes<true>, n);
        k_ray_lanes<true><<<gl, kQBlock, 0, stream>>>(n, order, ro, rd, pos, fid, depth, nodes, tris, lanes,
                                                      ctr + kCtRayLanesN, ctr + kCtRayLanesNext); count_launch();
    } else {
        const unsigned gl = persistent_grid(k_ray_lanes<false>, n);
        k_ray_lanes<false><<<gl, kQBlock, 0, stream>>>(n, order, ro, rd, pos, fid, depth, nodes, tris, lanes,
                                                       ctr + kCtRayLanesN, ctr + kCtRayLanesNext); count_launch();
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------ arena
// Query -> mesh: binary search over the meshes' first query indices.
__device__ __forceinline__ int mesh_of(const int64_t* __restrict__ qoff, int M, int64_t i) {
    int lo = 0, hi = M - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (qoff[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ uint32_t arena_cell(float3 p, const ArenaSortDesc& s) {
    const float side = (float)(1 << s.bits), m = side - 1.f;
    const float c[3] = {p.x, p.y, p.z};
    uint32_t g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float sc = s.hi[k] > s.lo[k] ? side / (s.hi[k] - s.lo[k]) : 0.f;
        const float v = (c[k] - s.lo[k]) * sc;
        g[k] = (uint32_t)fminf(fmaxf(v == v ? v : 0.f, 0.f), m);
    }
    return (uint32_t)s.cell_off + (spread3(g[0]) | (spread3(g[1]) << 1) | (spread3(g[2]) << 2));
}
__global__ void k_arena_hist(int64_t n, const float* __restrict__ pts, const int64_t* __restrict__ qoff, int M,
                             const ArenaSortDesc* __restrict__ sd, uint32_t* __restrict__ hist) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        atomicAdd(&hist[arena_cell(load3(pts, i), sd[mesh_of(qoff, M, i)])], 1u);
}
__global__ void k_arena_scatter(int64_t n, const float* __restrict__ pts, const int64_t* __restrict__ qoff, int M,
                                const ArenaSortDesc* __restrict__ sd, uint32_t* __restrict__ offs,
                                uint32_t* __restrict__ order) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        order[atomicAdd(&offs[arena_cell(load3(pts, i), sd[mesh_of(qoff, M, i)])], 1u)] = (uint32_t)i;
}

cudaError_t launch_arena_distance(const ArenaLaunch& a, const float* pts, float* dist, int64_t* fid, float* uvw,
                                  cudaStream_t stream) {
    if (a.n_queries <= 0) return cudaSuccess;
    const bool few = a.n_queries < kFewQueries;
    uint32_t* const order = few ? nullptr : a.order;
    cudaError_t e = cudaMemsetAsync(a.counters, 0, 256, stream);
    if (e != cudaSuccess) return e;
    if (!few) {
        if ((e = cudaMemsetAsync(a.hist, 0, sizeof(uint32_t) * (a.n_cells + 1), stream)) != cudaSuccess) return e;
        const unsigned g = (unsigned)sm_count() * 8;
        k_arena_hist<<<g, 256, 0, stream>>>(a.n_queries, pts, a.qoff, a.n_meshes, a.sort, a.hist); count_launch();
        scan::exclusive(a.hist, a.bsum, a.n_cells, stream);
        k_arena_scatter<<<g, 256, 0, stream>>>(a.n_queries, pts, a.qoff, a.n_meshes, a.sort, a.hist, a.order); count_launch();
    }
    const bool signed_any = a.n_wt_packets > 0 || a.n_rs_packets > 0;
    const Work all{a.packets, a.meshes, a.n_packets, 0};
    int32_t* const slots = signed_any ? a.slots : nullptr;
    if (few)
        launch_few(a.n_queries, pts, dist, fid, uvw, slots, a.tree, a.meshes, a.qoff, a.n_meshes, 0, stream);
    else
        launch_nearest(all, a.n_queries, order, pts, dist, fid, uvw, slots, a.tree, a.heavy, a.heavy_cap, a.counters, false,
                       stream);
    if (a.n_wt_packets > 0) {
        const Work w{a.wt_packets, a.meshes, a.n_wt_packets, 0};
        const unsigned gw = persistent_grid(k_sign_watertight<false>, 32 * a.n_wt_packets);
        k_sign_watertight<false><<<gw, kQBlock, 0, stream>>>(w, order, pts, dist, a.slots, a.tree.nodes, a.tree.tris,
                                                             a.tree.wtris, NearLists{}, nullptr, nullptr, a.counters + kCtSign,
                                                             grab_for(32 * a.n_wt_packets, gw), 0); count_launch();
    }
    if (a.n_rs_packets > 0) {
        const Work w{a.rs_packets, a.meshes, a.n_rs_packets, 0};
        if ((e = cudaMemsetAsync(a.parity, 0, sizeof(unsigned long long) * a.n_meshes, stream)) != cudaSuccess) return e;
        launch_raystab(w, 32 * a.n_rs_packets, order, pts, dist, a.tree.nodes, a.tree.tris, a.counters + kCtArenaRs,
                       a.rs_cand, a.counters + kCtCandN, a.counters + kCtLinesNext, a.tree.n_tris, a.face_off, a.face_slot,
                       a.n_meshes, a.parity, stream);
    }
    return cudaGetLastError();
}

int cell_bits_for(int64_t n) { return cell_bits(n); }

// The raystab stab directions of queries first .. first+n-1 (inspection):
// dirs[(i * 32 + k) * 3 + c], the same stab_dir values the sign pass uses.
__global__ void k_stab_dirs(int64_t n, uint32_t first, float* __restrict__ dirs) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 off = stab_offset(first + (uint32_t)i);
    float* o = dirs + i * 96;
    for (uint32_t k = 0; k < 32; ++k) {
        const float3 d = stab_dir(k, off);
        o[3 * k] = d.x;
        o[3 * k + 1] = d.y;
        o[3 * k + 2] = d.z;
    }
}

cudaError_t launch_stab_dirs(int64_t first, int64_t n, float* dirs, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    k_stab_dirs<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(n, (uint32_t)first, dirs); count_launch();
    return cudaGetLastError();
}

cudaError_t upload_constants() {
    float lat[64];
    const volatile float eps = 1.33f, phi = 1.6180339887498948482045868343656f;
    const float den = 31.0f + 2.0f * eps;
    for (int k = 0; k < 32; ++k) {
        lat[k] = ((float)k + eps) / den;
        lat[32 + k] = (float)k / phi;
    }
    return cudaMemcpyToSymbol(g_lattice, lat, sizeof(lat));
}

}  // namespace cubvh
