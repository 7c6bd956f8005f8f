// Sparse marching cubes: a triangle mesh of the iso-surface of per-voxel
// corner values over a sparse set of voxels.
//
// Reference: include/gpu/spcumc.cuh (`_sparse_marching_cubes`), entry
// cubvh/api.py:173-187.  Kept alike because they are the interface or decide
// the vertex array: the corner order of the [N, 8] input (offsets (0,0,0),
// (1,0,0), (1,1,0), (0,1,0), then the same at z + 1), the edge numbering
// (bottom square, top square, verticals), a corner is inside when its value
// is below iso, a vertex on every edge with one corner inside at
// t = clamp((iso - va) / (vb - va), 0, 1) (0.5 when |vb - va| < 1e-30) from
// the edge's first corner, vertices shared by voxels merged by their edge key
// (lower corner, axis) with the copy of the lowest voxel kept and the array
// sorted by key, and triangles listed voxel by voxel.  The optional corner
// averaging replaces every corner value by the mean over the voxels sharing
// that corner.
//
// Triangulation.  By default the reference's: each voxel's triangles come
// from the marching-cubes case table of its corner configuration (mc_cases.h,
// recovered from the reference's own outputs for the 256 configurations:
// tests/golden/make_ref_mc_cases.py), table triangle (e0, e1, e2) written as
// vertices (e0, e2, e1), voxel by voxel, so the triangle array equals the
// reference's index for index.  The table is the public marching-cubes case
// table; its configurations with faces cut four times (the ambiguous cases)
// are triangulated without looking at the face's saddle, so neighbouring
// cubes can disagree and leave holes there.
//
// Optionally (flag kSmcClosed) this file's own triangulation, no lookup
// table: on each cube face, walk its corners counter-clockwise as seen from
// outside the cube; a segment of the surface joins an edge where the walk
// enters the inside region to the next edge where it leaves it.  A face with
// four cut edges (inside corners on a diagonal) is resolved by the sign of
// its bilinear saddle (Nielson and Hamann's asymptotic decider): the two
// inside corners are joined through the face when the saddle value is below
// iso.  Both cubes sharing a face take the same decision, so the surface is
// closed wherever the corner values agree.  Every cut edge is entered on one
// of its faces and left on the other, so the segments form closed loops.
// Each loop, started at its lowest edge, is cut into a triangle fan from the
// first vertex none of whose diagonals joins two edges of one face that the
// loop crosses twice (such a diagonal would lie in that face and be shared
// with the neighbouring cube's triangles); when no vertex qualifies, ears
// whose closing diagonal avoids such faces are clipped one by one.
// Triangles face from the inside (values below iso) to the outside.  A cube
// with one corner inside gives the same triangle as the table.
#include <cstddef>
#include <cstdint>
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <mutex>
#include <string>
#include <vector>

#include "launches.h"
#include "kernels.h"
#include "mc_cases.h"
#include "scan.cuh"

namespace cubvh {
namespace {

__constant__ int8_t c_corner_off[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                          {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ int8_t c_edge_corners[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                             {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
// Faces: corners counter-clockwise seen from outside the cube, and the edge
// from corner i to corner i + 1 of that cycle.
__constant__ int8_t c_face_corners[6][4] = {{0, 3, 2, 1}, {4, 5, 6, 7}, {0, 1, 5, 4},
                                            {3, 7, 6, 2}, {0, 4, 7, 3}, {1, 2, 6, 5}};
__constant__ int8_t c_face_edges[6][4] = {{3, 2, 1, 0}, {4, 5, 6, 7}, {0, 9, 4, 8},
                                          {11, 6, 10, 2}, {8, 7, 11, 3}, {1, 10, 5, 9}};

struct Cube {
    float v[8];
    uint32_t inside;  // bit c: corner c below iso
    uint32_t cut;     // bit e: edge e has one corner inside
};

__device__ __forceinline__ Cube load_cube(const float* __restrict__ corners, int64_t i, float iso) {
    Cube c;
    c.inside = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        c.v[k] = corners[8 * i + k];
        if (c.v[k] < iso) c.inside |= 1u << k;
    }
    c.cut = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e)
        if (((c.inside >> c_edge_corners[e][0]) ^ (c.inside >> c_edge_corners[e][1])) & 1u) c.cut |= 1u << e;
    return c;
}

// True when the bilinear interpolant of a face with inside corners on one
// diagonal has its saddle below iso (the inside corners are joined across
// the face).  a, c and b, d are the two diagonals in cycle order.  Rounded
// operations only (no contraction): swapping the diagonals negates numerator
// and denominator exactly, so the two cubes sharing the face agree.
__device__ __forceinline__ bool saddle_inside(float a, float b, float c, float d, float iso) {
    const float num = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, d));
    const float den = __fsub_rn(__fadd_rn(a, c), __fadd_rn(b, d));
    const float lim = __fmul_rn(iso, den);
    if (den > 0.f) return num < lim;
    if (den < 0.f) return num > lim;
    return false;  // flat saddle: keep the inside corners apart
}

// nxt[e] for every cut edge e: the edge the surface loop goes to after e.
__device__ __forceinline__ void surface_links(const Cube& c, float iso, int8_t nxt[12]) {
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        bool in[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) in[i] = (c.inside >> c_face_corners[f][i]) & 1u;
        int crossings = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) crossings += in[i] != in[(i + 1) & 3];
        if (crossings == 0) continue;
        bool join_inside = false;  // four crossings: are the inside corners joined?
        if (crossings == 4)
            join_inside = saddle_inside(c.v[c_face_corners[f][0]], c.v[c_face_corners[f][1]],
                                        c.v[c_face_corners[f][2]], c.v[c_face_corners[f][3]], iso);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int ip = (i + 3) & 3;  // previous corner in the cycle
            const int e_before = c_face_edges[f][ip], e_after = c_face_edges[f][i];
            if (crossings == 2) {
                // the inside run starts at the corner after the in-edge
                if (in[i] && !in[ip]) {
                    int j = i;
                    while (in[(j + 1) & 3]) j = (j + 1) & 3;
                    nxt[e_before] = c_face_edges[f][j];
                }
            } else if (join_inside) {
                // segments around the outside corners: in-edge after it -> out-edge before it
                if (!in[i]) nxt[e_after] = e_before;
            } else {
                // segments around the inside corners: in-edge before it -> out-edge after it
                if (in[i]) nxt[e_before] = e_after;
            }
        }
    }
}

__device__ __forceinline__ int n_triangles(const Cube& c, float iso) {
    if (!c.cut) return 0;
    int8_t nxt[12];
    surface_links(c, iso, nxt);
    uint32_t left = c.cut;
    int loops = 0;
    // nxt is a permutation of the cut edges (each is entered on one of its
    // faces and left on the other): the walks close; 12 steps bound them all
    int steps = 0;
    while (left && steps < 12) {
        const int s = __ffs(left) - 1;
        int e = s;
        do { left &= ~(1u << e); e = nxt[e]; ++steps; } while (e != s && steps < 12);
        ++loops;
    }
    return __popc(c.cut) - 2 * loops;
}

// triangles of a corner configuration in the case table
__device__ __forceinline__ int n_table_triangles(uint32_t inside) {
    int t = 0;
    while (t < 5 && c_mc_tri[inside][3 * t] >= 0) ++t;
    return t;
}

// Bound: launches and host round trips.  The surface voxels of a 192^3 grid
// (22 MB of inputs and results: 3.4 us of memory time) take about 105 us of
// kernels, 52 of them the radix sort's, and three waits (the counts, the
// merged vertices, the release).  So few launches: the count kernel takes the
// coordinate bounds along, count and emit scan their own block's counts (a
// prefix over all voxels is one small launch between them), emit writes the
// sort's values, merge scans its own run starts; two workspaces instead of
// twenty allocations; and keys of the smallest type and bit count that hold
// the range.  213 us a call against 333 with separate bounds, scans, index
// and head passes and 26-bit keys in 64 bits.
constexpr int kSmcBlock = 256;
struct SmcTotals { int32_t lo[3], hi[3]; uint32_t nv, nt; };   // coordinate bounds, vertices, triangles

// Exclusive prefix of v over the block's threads; every thread gets the total.
__device__ __forceinline__ uint32_t smc_block_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t s_warp[kSmcBlock / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kSmcBlock / 32; ++k) {
        before += k < w ? s_warp[k] : 0u;
        all += s_warp[k];
    }
    *total = all;
    return before + inc - v;
}

// Per voxel its vertices (low byte) and triangles (high byte); per block their
// sums and the coordinate bounds.
__global__ void __launch_bounds__(kSmcBlock) k_smc_count(int64_t n, const int32_t* __restrict__ coords,
                                                         const float* __restrict__ corners, float iso, bool table,
                                                         uint16_t* __restrict__ counts, uint2* __restrict__ bsum,
                                                         int32_t* __restrict__ bbox) {
    const int64_t i = (int64_t)blockIdx.x * kSmcBlock + threadIdx.x;
    int lo[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, hi[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    uint32_t nv = 0, nt = 0;
    if (i < n) {
        const Cube c = load_cube(corners, i, iso);
        nv = __popc(c.cut);
        nt = (uint32_t)(table ? n_table_triangles(c.inside) : n_triangles(c, iso));
        counts[i] = (uint16_t)(nv | (nt << 8));
#pragma unroll
        for (int k = 0; k < 3; ++k) lo[k] = hi[k] = coords[3 * i + k];
    }
    __shared__ int32_t sb[6];
    if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? INT32_MAX : INT32_MIN;
    uint32_t total;
    smc_block_scan(nv | (nt << 16), &total);   // at most 12 * 256 each
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = __reduce_min_sync(0xFFFFFFFFu, lo[k]);
        hi[k] = __reduce_max_sync(0xFFFFFFFFu, hi[k]);
    }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) { atomicMin(&sb[k], lo[k]); atomicMax(&sb[3 + k], hi[k]); }
    __syncthreads();
    if (threadIdx.x == 0) bsum[blockIdx.x] = make_uint2(total & 0xFFFFu, total >> 16);
    if (threadIdx.x < 6) bbox[6 * (int64_t)blockIdx.x + threadIdx.x] = sb[threadIdx.x];
}
// One block: exclusive prefixes of the block sums, totals and bounds.
__global__ void __launch_bounds__(1024) k_smc_top(int64_t nblk, const uint2* __restrict__ bsum,
                                                  const int32_t* __restrict__ bbox, uint2* __restrict__ bpre,
                                                  SmcTotals* __restrict__ out) {
    __shared__ uint2 sh[1024];
    __shared__ int32_t sb[6];
    if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? INT32_MAX : INT32_MIN;
    __syncthreads();
    const int64_t per = (nblk + 1023) / 1024;
    const int64_t b0 = threadIdx.x * per, b1 = min(b0 + per, nblk);
    uint2 s = make_uint2(0u, 0u);
#pragma unroll 8
    for (int64_t i = b0; i < b1; ++i) { s.x += bsum[i].x; s.y += bsum[i].y; }
    int v[6] = {INT32_MAX, INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN, INT32_MIN};
    for (int64_t i = threadIdx.x; i < nblk; i += 1024)
#pragma unroll
        for (int k = 0; k < 3; ++k) { v[k] = min(v[k], bbox[6 * i + k]); v[3 + k] = max(v[3 + k], bbox[6 * i + 3 + k]); }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[k] = __reduce_min_sync(0xFFFFFFFFu, v[k]);
        v[3 + k] = __reduce_max_sync(0xFFFFFFFFu, v[3 + k]);
    }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) { atomicMin(&sb[k], v[k]); atomicMax(&sb[3 + k], v[3 + k]); }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const uint2 t = threadIdx.x >= (unsigned)o ? sh[threadIdx.x - o] : make_uint2(0u, 0u);
        __syncthreads();
        sh[threadIdx.x].x += t.x;
        sh[threadIdx.x].y += t.y;
        __syncthreads();
    }
    uint2 run = threadIdx.x ? sh[threadIdx.x - 1] : make_uint2(0u, 0u);
#pragma unroll 8
    for (int64_t i = b0; i < b1; ++i) {
        const uint2 t = bsum[i];
        bpre[i] = run;
        run.x += t.x;
        run.y += t.y;
    }
    if (threadIdx.x < 3) { out->lo[threadIdx.x] = sb[threadIdx.x]; out->hi[threadIdx.x] = sb[3 + threadIdx.x]; }
    if (threadIdx.x == 1023) { out->nv = sh[1023].x; out->nt = sh[1023].y; }
}

struct KeyPack {
    int32_t minx, miny, minz;
    uint64_t ry, rz;  // extents (in corners) along y and z
};
__device__ __forceinline__ uint64_t pack_point(int x, int y, int z, const KeyPack& k) {
    return ((uint64_t)(uint32_t)(x - k.minx) * k.ry + (uint64_t)(uint32_t)(y - k.miny)) * k.rz +
           (uint64_t)(uint32_t)(z - k.minz);
}

// Vertices (position, edge key) in edge order and triangles (indices into
// this launch's vertex list, before merging) of every voxel.
template <class Key>
__global__ void __launch_bounds__(kSmcBlock, 4) k_smc_emit(int64_t n, const int32_t* __restrict__ coords,
                           const float* __restrict__ corners, float iso, bool table,
                           const uint16_t* __restrict__ counts, const uint2* __restrict__ bpre, KeyPack kp,
                           float* __restrict__ pos, Key* __restrict__ key, int32_t* __restrict__ ord,
                           int32_t* __restrict__ tri) {
    const int64_t i = (int64_t)blockIdx.x * kSmcBlock + threadIdx.x;
    const uint32_t mine = i < n ? counts[i] : 0u;
    uint32_t total;
    const uint32_t before = smc_block_scan((mine & 0xFFu) | ((mine >> 8) << 16), &total);
    if (mine) {
        const uint2 base = bpre[blockIdx.x];
        const Cube c = load_cube(corners, i, iso);
        const int x = coords[3 * i], y = coords[3 * i + 1], z = coords[3 * i + 2];
        const uint32_t vb = base.x + (before & 0xFFFFu);
        uint32_t k = vb;
        for (int e = 0; e < 12; ++e) {
            if (!((c.cut >> e) & 1u)) continue;
            const int a = c_edge_corners[e][0], b = c_edge_corners[e][1];
            const float va = c.v[a], vv = c.v[b];
            const float den = __fsub_rn(vv, va);
            float t;
            if (fabsf(den) < 1e-30f) {
                t = 0.5f;
            } else {
                t = __fdiv_rn(__fsub_rn(iso, va), den);
                t = fminf(fmaxf(t, 0.f), 1.f);
            }
            const int ax = x + c_corner_off[a][0], ay = y + c_corner_off[a][1], az = z + c_corner_off[a][2];
            const int bx = x + c_corner_off[b][0], by = y + c_corner_off[b][1], bz = z + c_corner_off[b][2];
            pos[3 * (int64_t)k] = __fmaf_rn(t, __fsub_rn((float)bx, (float)ax), (float)ax);
            pos[3 * (int64_t)k + 1] = __fmaf_rn(t, __fsub_rn((float)by, (float)ay), (float)ay);
            pos[3 * (int64_t)k + 2] = __fmaf_rn(t, __fsub_rn((float)bz, (float)az), (float)az);
            const int axis = ax != bx ? 0 : (ay != by ? 1 : 2);
            key[k] = (Key)(pack_point(min(ax, bx), min(ay, by), min(az, bz), kp) * 3u + (uint64_t)axis);
            ord[k] = (int32_t)k;
            ++k;
        }
        uint32_t t_out = base.y + (before >> 16);
        const uint32_t t_end = t_out + (mine >> 8);  // the count pass's triangles: never write past them
        auto vid = [&](int e) { return (int32_t)(vb + __popc(c.cut & ((1u << e) - 1u))); };
        if (table) {
            // the case table's triangles, written (e0, e2, e1) as the reference does
            for (int t = 0; t < 5 && t_out < t_end; ++t) {
                const int e0 = c_mc_tri[c.inside][3 * t];
                if (e0 < 0) break;
                tri[3 * (int64_t)t_out] = vid(e0);
                tri[3 * (int64_t)t_out + 1] = vid(c_mc_tri[c.inside][3 * t + 2]);
                tri[3 * (int64_t)t_out + 2] = vid(c_mc_tri[c.inside][3 * t + 1]);
                ++t_out;
            }
            return;
        }
        int8_t nxt[12];
        surface_links(c, iso, nxt);
        // loops, in order of their lowest edge
        int8_t loop_of[12];
        int8_t seq[12];
        int8_t start[7];
        int nl = 0, len = 0;
        {
            uint32_t left = c.cut;
            while (left && nl < 6 && len < 12) {
                const int s0 = __ffs(left) - 1;
                start[nl] = (int8_t)len;
                int e = s0;
                do { left &= ~(1u << e); loop_of[e] = (int8_t)nl; seq[len++] = (int8_t)e; e = nxt[e]; }
                while (e != s0 && len < 12);
                ++nl;
            }
            start[nl] = (int8_t)len;
        }
        // mark[e]: faces with four cut edges whose two segments both lie in e's
        // loop; two such vertices not joined by a segment must not be joined by
        // a diagonal either (it would lie in the face, and the neighbouring cube
        // could use it too)
        uint8_t mark[12];
#pragma unroll
        for (int e = 0; e < 12; ++e) mark[e] = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            const int e0 = c_face_edges[f][0], e1 = c_face_edges[f][1], e2 = c_face_edges[f][2],
                      e3 = c_face_edges[f][3];
            if (((c.cut >> e0) & (c.cut >> e1) & (c.cut >> e2) & (c.cut >> e3) & 1u) &&
                loop_of[e0] == loop_of[e1] && loop_of[e1] == loop_of[e2] && loop_of[e2] == loop_of[e3]) {
                mark[e0] |= 1u << f; mark[e1] |= 1u << f; mark[e2] |= 1u << f; mark[e3] |= 1u << f;
            }
        }
        for (int l = 0; l < nl && t_out < t_end; ++l) {
            const int b0 = start[l], L = start[l + 1] - start[l];
            int8_t* q = seq + b0;
            // fan apex: the first vertex none of whose diagonals joins two
            // vertices of one marked face
            int apex = -1;
            for (int k = 0; k < L && apex < 0; ++k) {
                bool ok = true;
                for (int j = 0; j < L && ok; ++j) {
                    const int dj = (j - k + L) % L;
                    if (dj <= 1 || dj == L - 1) continue;
                    if (mark[q[k]] & mark[q[j]]) ok = false;
                }
                if (ok) apex = k;
            }
            if (apex >= 0) {
                for (int m = 1; m + 1 < L && t_out < t_end; ++m) {
                    tri[3 * (int64_t)t_out] = vid(q[apex]);
                    tri[3 * (int64_t)t_out + 1] = vid(q[(apex + m) % L]);
                    tri[3 * (int64_t)t_out + 2] = vid(q[(apex + m + 1) % L]);
                    ++t_out;
                }
            } else {
                // ear clipping: cut the first ear whose new edge is allowed (any
                // ear if none is), keeping the loop's orientation
                int8_t ring[12];
                for (int m = 0; m < L; ++m) ring[m] = q[m];
                int r = L;
                while (r >= 3 && t_out < t_end) {
                    int ear = 1;
                    for (int m = 0; m < r; ++m) {
                        const int a0 = ring[(m + r - 1) % r], a2 = ring[(m + 1) % r];
                        if (r == 3 || !(mark[a0] & mark[a2])) { ear = m; break; }
                    }
                    tri[3 * (int64_t)t_out] = vid(ring[(ear + r - 1) % r]);
                    tri[3 * (int64_t)t_out + 1] = vid(ring[ear]);
                    tri[3 * (int64_t)t_out + 2] = vid(ring[(ear + 1) % r]);
                    ++t_out;
                    for (int m = ear; m + 1 < r; ++m) ring[m] = ring[m + 1];
                    --r;
                }
            }
        }
    }
}


// sorted keys: the runs that start in each block
template <class Key>
__global__ void __launch_bounds__(kSmcBlock) k_smc_heads(int64_t m, const Key* __restrict__ key,
                                                         uint32_t* __restrict__ hsum) {
    const int64_t i = (int64_t)blockIdx.x * kSmcBlock + threadIdx.x;
    const int c = __syncthreads_count(i < m && (i == 0 || key[i] != key[i - 1]));
    if (threadIdx.x == 0) hsum[blockIdx.x] = (uint32_t)c;
}
// hsum: exclusive prefixes of the blocks' run starts; the run's first (lowest
// emission index, the sort being stable) supplies the merged vertex's position
template <class Key>
__global__ void __launch_bounds__(kSmcBlock) k_smc_merge(int64_t m, const Key* __restrict__ key,
                            const uint32_t* __restrict__ hsum, const int32_t* __restrict__ order,
                            const float* __restrict__ pos, int32_t* __restrict__ map, float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * kSmcBlock + threadIdx.x;
    const uint32_t head = i < m && (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
    uint32_t total;
    const uint32_t before = smc_block_scan(head, &total);
    if (i >= m) return;
    const int32_t id = (int32_t)(hsum[blockIdx.x] + before + head) - 1;
    const int32_t src = order[i];
    map[src] = id;
    if (head) {
        const int64_t to = 3 * (int64_t)id, from = 3 * (int64_t)src;
        out[to] = pos[from];
        out[to + 1] = pos[from + 1];
        out[to + 2] = pos[from + 2];
    }
}
__global__ void k_smc_remap(int64_t n3, const int32_t* __restrict__ map, int32_t* __restrict__ tri) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += (int64_t)gridDim.x * blockDim.x)
        tri[i] = map[tri[i]];
}

// corner averaging: keys of the 8 corners of every voxel
template <class Key>
__global__ void k_smc_corner_keys(int64_t n, const int32_t* __restrict__ coords, KeyPack kp, Key* __restrict__ key,
                                  int32_t* __restrict__ idx) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < 8 * n; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = j >> 3;
        const int c = (int)(j & 7);
        key[j] = (Key)pack_point(coords[3 * i] + c_corner_off[c][0], coords[3 * i + 1] + c_corner_off[c][1],
                                 coords[3 * i + 2] + c_corner_off[c][2], kp);
        idx[j] = (int32_t)j;
    }
}
// one thread per run of equal corner keys: the mean of the run's values, in
// run order (voxel order), written back to every member
template <class Key>
__global__ void k_smc_corner_mean(int64_t m, const Key* __restrict__ key, const int32_t* __restrict__ idx,
                                  const float* __restrict__ in, float* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        if (i > 0 && key[i] == key[i - 1]) continue;
        float sum = 0.f;
        int cnt = 0;
        int64_t j = i;
        do { sum = __fadd_rn(sum, in[idx[j]]); ++cnt; ++j; } while (j < m && key[j] == key[i]);
        const float mean = __fdiv_rn(sum, (float)cnt);
        for (int64_t q = i; q < j; ++q) out[idx[q]] = mean;
    }
}

unsigned grid_for(int64_t n) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = (n + 255) / 256;
    const int64_t cap = (int64_t)nsm * 16;
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

int bits_for(uint64_t v) {  // bits to hold values below v
    int b = 0;
    while (b < 64 && (uint64_t(1) << b) < v) ++b;
    return b;
}

template <class T>
cudaError_t pool_get(cudaMemPool_t pool, cudaStream_t s, T** out, size_t count) {
    void* q = nullptr;
    const cudaError_t e = cudaMallocFromPoolAsync(&q, count * sizeof(T) > 0 ? count * sizeof(T) : 16, pool, s);
    if (e == cudaSuccess) *out = static_cast<T*>(q);
    return e;
}

// Stream-ordered temporaries of one call: every buffer taken from `get` is
// returned with cudaFreeAsync on the same stream, early through `put` or at
// scope exit, so an error return in the middle of the pipeline leaks nothing.
struct AsyncTemps {
    cudaMemPool_t pool;
    cudaStream_t s;
    std::vector<void*> p;
    AsyncTemps(cudaMemPool_t pl, cudaStream_t st) : pool(pl), s(st) {}
    AsyncTemps(const AsyncTemps&) = delete;
    AsyncTemps& operator=(const AsyncTemps&) = delete;
    ~AsyncTemps() { for (void* q : p) cudaFreeAsync(q, s); }
    template <class T>
    cudaError_t get(T** out, size_t count) {
        const cudaError_t e = pool_get(pool, s, out, count);
        if (e == cudaSuccess) p.push_back(*out);
        return e;
    }
    void put(void* q) {
        for (size_t i = 0; i < p.size(); ++i)
            if (p[i] == q) { cudaFreeAsync(q, s); p.erase(p.begin() + (std::ptrdiff_t)i); return; }
    }
};

// Several arrays in one allocation: the places first, the pointers once it is made.
struct Layout {
    size_t bytes = 0;
    template <class T>
    size_t add(size_t count) {
        const size_t at = bytes;
        bytes += (count * sizeof(T) + 255) & ~size_t(255);
        return at;
    }
};

// Every corner's mean over the voxels that share it, by a sort of all corners.
template <class Key>
int smc_average(int64_t n, const int32_t* coords, const float* corners, KeyPack kp, int cbits, AsyncTemps& tmp,
                cudaStream_t s, float* avg, std::string& err) {
    cudaError_t e;
    auto fail = [&](cudaError_t x, const char* what) { err = std::string(what) + ": " + cudaGetErrorString(x); return 2; };
    const int64_t m = 8 * n;
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (Key*)nullptr, (Key*)nullptr, (int32_t*)nullptr, (int32_t*)nullptr,
                                    (int)m, 0, cbits, s);
    Layout lay;
    const size_t o_key = lay.add<Key>(m), o_key2 = lay.add<Key>(m), o_idx = lay.add<int32_t>(m),
                 o_idx2 = lay.add<int32_t>(m), o_sort = lay.add<char>(tb);
    char* ws = nullptr;
    if ((e = tmp.get(&ws, lay.bytes)) != cudaSuccess) return fail(e, "pool allocation");
    Key *key = reinterpret_cast<Key*>(ws + o_key), *key2 = reinterpret_cast<Key*>(ws + o_key2);
    int32_t *idx = reinterpret_cast<int32_t*>(ws + o_idx), *idx2 = reinterpret_cast<int32_t*>(ws + o_idx2);
    k_smc_corner_keys<Key><<<grid_for(m), 256, 0, s>>>(n, coords, kp, key, idx); count_launch();
    if ((e = cub::DeviceRadixSort::SortPairs(ws + o_sort, tb, key, key2, idx, idx2, (int)m, 0, cbits, s)) != cudaSuccess)
        return fail(e, "corner sort");
    count_launch();
    k_smc_corner_mean<Key><<<grid_for(m), 256, 0, s>>>(m, key2, idx2, corners, avg); count_launch();
    tmp.put(ws);
    return 0;
}

// Vertices and triangles of the m cut edges and t triangles counted: emission,
// merge by edge key (Key: the smallest type that holds key_bits), remapping.
template <class Key>
int smc_vertices(int64_t n, const int32_t* coords, const float* use, float iso, bool table, const uint16_t* counts,
                 const uint2* bpre, KeyPack kp, int key_bits, int64_t m, int64_t t, AsyncTemps& tmp, cudaStream_t s,
                 SparseMCResult& out, std::string& err) {
    cudaError_t e;
    auto fail = [&](cudaError_t x, const char* what) { err = std::string(what) + ": " + cudaGetErrorString(x); return 2; };
    const unsigned gm = (unsigned)((m + kSmcBlock - 1) / kSmcBlock);
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (Key*)nullptr, (Key*)nullptr, (int32_t*)nullptr, (int32_t*)nullptr,
                                    (int)m, 0, key_bits, s);
    Layout lay;
    const size_t o_pos = lay.add<float>(3 * m), o_key = lay.add<Key>(m), o_key2 = lay.add<Key>(m),
                 o_ord = lay.add<int32_t>(m), o_ord2 = lay.add<int32_t>(m), o_map = lay.add<int32_t>(m),
                 o_hsum = lay.add<uint32_t>((size_t)gm + 1), o_sort = lay.add<char>(tb);
    char* ws = nullptr;
    if ((e = tmp.get(&ws, lay.bytes)) != cudaSuccess) return fail(e, "sparse marching cubes buffers");
    float* pos = reinterpret_cast<float*>(ws + o_pos);
    Key *key = reinterpret_cast<Key*>(ws + o_key), *key2 = reinterpret_cast<Key*>(ws + o_key2);
    int32_t *ord = reinterpret_cast<int32_t*>(ws + o_ord), *ord2 = reinterpret_cast<int32_t*>(ws + o_ord2),
            *map = reinterpret_cast<int32_t*>(ws + o_map);
    uint32_t* hsum = reinterpret_cast<uint32_t*>(ws + o_hsum);
    const unsigned g = (unsigned)((n + kSmcBlock - 1) / kSmcBlock);
    k_smc_emit<Key><<<g, kSmcBlock, 0, s>>>(n, coords, use, iso, table, counts, bpre, kp, pos, key, ord, out.tris);
    count_launch();
    // the emission index as the value: the stable sort keeps each key's lowest first
    if ((e = cub::DeviceRadixSort::SortPairs(ws + o_sort, tb, key, key2, ord, ord2, (int)m, 0, key_bits, s)) != cudaSuccess)
        return fail(e, "edge key sort");
    count_launch();
    k_smc_heads<Key><<<gm, kSmcBlock, 0, s>>>(m, key2, hsum); count_launch();
    scan::k_top<<<1, 1024, 0, s>>>(hsum, (int64_t)gm); count_launch();   // hsum[gm] = merged vertex count
    uint32_t u = 0;
    if ((e = cudaMemcpyAsync(&u, hsum + gm, sizeof(uint32_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return fail(e, "sparse marching cubes merge");
    if ((e = pool_get(tmp.pool, s, &out.verts, (size_t)3 * u)) != cudaSuccess) return fail(e, "vertex buffer");
    k_smc_merge<Key><<<gm, kSmcBlock, 0, s>>>(m, key2, hsum, ord2, pos, map, out.verts); count_launch();
    if (t > 0) { k_smc_remap<<<grid_for(3 * t), 256, 0, s>>>(3 * t, map, out.tris); count_launch(); }
    out.n_verts = u;
    out.n_tris = t;
    return 0;
}

}  // namespace

// Temporaries and results come from the library's pool on `stream`; the
// results stay in `out` (owned by the caller through cubvh_sparse_mc_*,
// which releases them on an error return as well).
int sparse_mc_run(const int32_t* coords, const float* corners, int64_t n, float iso, bool ensure_consistency,
                  bool closed, cudaStream_t s, SparseMCResult& out, std::string& err) {
    out = SparseMCResult{};
    if (n <= 0) return 0;
    if (n > (int64_t)INT32_MAX / 12) { err = "too many voxels (the vertex count must fit in int32)"; return 1; }
    cudaError_t e;
    auto fail = [&](cudaError_t x, const char* what) { err = std::string(what) + ": " + cudaGetErrorString(x); return 2; };
    cudaMemPool_t pool = nullptr;
    if ((e = library_pool(&pool)) != cudaSuccess) return fail(e, "memory pool");
    AsyncTemps tmp(pool, s);
    const unsigned g = (unsigned)((n + kSmcBlock - 1) / kSmcBlock);
    Layout lay;
    const size_t o_counts = lay.add<uint16_t>(n), o_bsum = lay.add<uint2>(g), o_bpre = lay.add<uint2>(g),
                 o_bbox = lay.add<int32_t>(6 * (size_t)g), o_tot = lay.add<SmcTotals>(1);
    char* ws = nullptr;
    if ((e = tmp.get(&ws, lay.bytes)) != cudaSuccess) return fail(e, "pool allocation");
    uint16_t* counts = reinterpret_cast<uint16_t*>(ws + o_counts);
    uint2 *bsum = reinterpret_cast<uint2*>(ws + o_bsum), *bpre = reinterpret_cast<uint2*>(ws + o_bpre);
    int32_t* bbox = reinterpret_cast<int32_t*>(ws + o_bbox);
    SmcTotals* d_tot = reinterpret_cast<SmcTotals*>(ws + o_tot);
    // counts, their block prefixes and the coordinate bounds (host round trip)
    SmcTotals tot{};
    auto count = [&](const float* from) {
        k_smc_count<<<g, kSmcBlock, 0, s>>>(n, coords, from, iso, !closed, counts, bsum, bbox); count_launch();
        k_smc_top<<<1, 1024, 0, s>>>(g, bsum, bbox, bpre, d_tot); count_launch();
        const cudaError_t x = cudaMemcpyAsync(&tot, d_tot, sizeof(tot), cudaMemcpyDeviceToHost, s);
        return x == cudaSuccess ? cudaStreamSynchronize(s) : x;
    };
    if ((e = count(corners)) != cudaSuccess) return fail(e, "sparse marching cubes counts");
    const uint64_t rx = (uint64_t)((int64_t)tot.hi[0] - tot.lo[0] + 2), ry = (uint64_t)((int64_t)tot.hi[1] - tot.lo[1] + 2),
                   rz = (uint64_t)((int64_t)tot.hi[2] - tot.lo[2] + 2);
    if (bits_for(rx) + bits_for(ry) + bits_for(rz) + 2 > 64) {
        err = "voxel coordinate range too large for 64-bit edge keys";
        return 1;
    }
    // the keys are mixed-radix numbers below this: 24 bits (three sort passes)
    // where bits per coordinate make 26 (four) for a 167^3 range
    const int key_bits = bits_for(rx * ry * rz * 3);
    const KeyPack kp{tot.lo[0], tot.lo[1], tot.lo[2], ry, rz};

    const float* use = corners;
    if (ensure_consistency) {
        float* avg = nullptr;
        if ((e = tmp.get(&avg, 8 * n)) != cudaSuccess) return fail(e, "pool allocation");
        const int cbits = bits_for(rx * ry * rz);
        const int rc = cbits <= 32 ? smc_average<uint32_t>(n, coords, corners, kp, cbits, tmp, s, avg, err)
                                   : smc_average<uint64_t>(n, coords, corners, kp, cbits, tmp, s, avg, err);
        if (rc != 0) return rc;
        use = avg;  // freed at scope exit, after the kernels that read it
        if ((e = count(avg)) != cudaSuccess) return fail(e, "sparse marching cubes counts");
    }
    const int64_t m = tot.nv, t = tot.nt;
    if (m > 0) {
        if ((e = pool_get(pool, s, &out.tris, (size_t)(3 * t))) != cudaSuccess) return fail(e, "sparse marching cubes buffers");
        const int rc = key_bits <= 32
            ? smc_vertices<uint32_t>(n, coords, use, iso, !closed, counts, bpre, kp, key_bits, m, t, tmp, s, out, err)
            : smc_vertices<uint64_t>(n, coords, use, iso, !closed, counts, bpre, kp, key_bits, m, t, tmp, s, out, err);
        if (rc != 0) return rc;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "sparse marching cubes launch");
    return 0;
}

// The caller has waited for every stream that used the buffers (host-side),
// so the frees need no ordering: the per-thread stream takes them.
void sparse_mc_release(SparseMCResult& r) {
    if (r.verts) cudaFreeAsync(r.verts, cudaStreamPerThread);
    if (r.tris) cudaFreeAsync(r.tris, cudaStreamPerThread);
    r = SparseMCResult{};
}

}  // namespace cubvh
