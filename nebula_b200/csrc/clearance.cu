// Clearance map: where in the domain a short straight step cannot meet a
// triangle.
//
// Nearly all transport steps are short (half of them below 0.4 nm) and end
// inside one material: on the benchmark scans only 1-3 % of the steps meet a
// triangle, yet every step used to walk the octree leaf it starts in (about
// ten triangles).  The map answers most of them with two gathers.
//
// Layout: a coarse grid of cells over the octree's root box, each either
// empty (nothing within `reach`, or within `far_reach`) or the index of a
// brick of 4 x 4 x 4 records, one per fine cell of edge h.  A record is two
// slabs: every part of every triangle inside the fine cell's box, widened by
// `reach` on all sides, lies within |n . q - c| <= 1 of one of them, where q
// is the position relative to the fine cell's centre and n the slab's normal
// divided by its half thickness (a margin for rounding included).  A step
// shorter than `reach` stays inside the widened box, so when its two ends lie
// on the same side of the one slab and on the same side of the other it meets
// no triangle.  Surfaces are locally flat, so a slab is thin (only the
// margin, on flat faces); the second one serves edges and corners.
//
// The margin covers the rounding of the exact test, because "meets no
// triangle" has to mean that intersect_ray reports no hit.  With u = 2^-24,
// |s| the distance from the triangle's corner to the ray's start and k =
// |e1||e2| / |e1 x e2|, the test's three numerators are off by at most
// 12 u |s| times the edges in them and its determinant by 8 u |e1||e2|, so the
// point that it reports lies within 44 u k |s| / cos of the triangle, cos being
// that of the ray's angle to the triangle's normal, and along that normal
// within 12 u k |s|.  A triangle's `slack` is 24 u k |s| plus the 2.4e-6 of its
// edges by which the test enlarges it; at an angle phi to its slab it widens
// the slab by slack / 2 + 10 slack sin(phi), which covers rays down to a cosine
// of 0.18 at the bound and of 0.02 at the errors that occur (a tenth of it),
// and it is a candidate of the cells within 10 slack.  Triangles of sound
// meshes mostly have a slack below 0.01 nm, and the margin decides; strips of
// 1000 nm x 0.3 nm (5 nm) make the cells round them walk.  With one margin for
// all shapes, runs through sheets of strips had 4 of 35,305 crossings fewer
// than the walk reports (4000 nm x 4 nm) and 247 of 28,966 (8000 nm x 1 nm).
//
// h = 4 nm and reach = 3 nm: 99 % of the free paths are below 3 nm.  Share of
// steps answered on 8,000-step samples (grating, rough slab, contact holes):
// 0.92 / 0.91 / 0.83 with two slabs, 0.84 / 0.91 / 0.68 with one; h = 2 adds
// 0.00 / 0.02 / 0.01 for eight times the records, h = 8 with a reach of 8 nm
// and one slab gives 0.52 / 0.82 / 0.32.
// B200, the second slab together with the walk's batched exact test: half the
// benchmark's grating frame 98.2 -> 80.3 ms, contact holes 41.0 -> 30.4 ms.
#include "clearance.h"

#include <algorithm>
#include <cmath>

#include "features.cuh"

namespace nbx {
namespace {

constexpr int kBrick = 4;            // fine cells per brick edge
constexpr int kBigCells = 4096;      // triangles over more coarse cells go to the grid-wide pass

struct Grid {
    float lox, loy, loz;   // root box corner
    float cell;            // coarse cell edge
    int nx, ny, nz;        // coarse cells
    float reach;           // widening of the boxes (margin included)
};

struct TriBox {
    float3 a, e1, e2, lo, hi;
    float3 u;      // unit normal (zero without an area)
    float slack;   // rounding of the exact test (nm; infinite without an area)
    float grow;    // boxes within this distance (nm) count as near
};

__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(a, fminf(b, c)); }
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(a, fmaxf(b, c)); }

// The normal is formed in double precision: that of a needle would be lost in
// single precision, and with it the plane test of near_box.
__device__ __forceinline__ TriBox load_tri(const float4* tri, int t, const Grid& g) {
    const float4 A = __ldg(tri + 3 * size_t(t)), B = __ldg(tri + 3 * size_t(t) + 1), C = __ldg(tri + 3 * size_t(t) + 2);
    TriBox r;
    r.a = make_float3(A.x, A.y, A.z);
    r.e1 = make_float3(B.x, B.y, B.z);
    r.e2 = make_float3(C.x, C.y, C.z);
    r.lo = make_float3(A.x + min3(0.0f, B.x, C.x), A.y + min3(0.0f, B.y, C.y), A.z + min3(0.0f, B.z, C.z));
    r.hi = make_float3(A.x + max3(0.0f, B.x, C.x), A.y + max3(0.0f, B.y, C.y), A.z + max3(0.0f, B.z, C.z));
    const double nx = double(B.y) * C.z - double(B.z) * C.y, ny = double(B.z) * C.x - double(B.x) * C.z,
                 nz = double(B.x) * C.y - double(B.y) * C.x;
    const double l2 = nx * nx + ny * ny + nz * nz;
    const double s = l2 > 0.0 ? rsqrt(l2) : 0.0;
    r.u = make_float3(float(nx * s), float(ny * s), float(nz * s));
    const float b2 = B.x * B.x + B.y * B.y + B.z * B.z, c2 = C.x * C.x + C.y * C.y + C.z * C.z;
    const float k = s > 0.0 ? sqrtf(b2) * sqrtf(c2) * float(s) : INFINITY;
    const float dx = r.hi.x - r.lo.x, dy = r.hi.y - r.lo.y, dz = r.hi.z - r.lo.z;
    const float size = sqrtf(dx * dx + dy * dy + dz * dz);   // at least the longest edge
    const float near = 1.75f * (g.cell / kBrick + 2.0f * g.reach);   // diagonal of a widened fine cell
    r.slack = 24.0f * 5.9604645e-8f * k * (size + near) + 2.4e-6f * size;
    r.grow = fminf(10.0f * r.slack, fminf(2.0f * size, 8.0f * g.cell));
    return r;
}

// Conservative triangle / box test: bounding boxes, then the triangle's
// plane against the box.  (cx, cy, cz) is the box centre, h its half edge.
__device__ __forceinline__ bool near_box(const TriBox& t, float cx, float cy, float cz, float h) {
    h += t.grow;
    if (t.lo.x > cx + h || t.hi.x < cx - h || t.lo.y > cy + h || t.hi.y < cy - h || t.lo.z > cz + h || t.hi.z < cz - h)
        return false;
    const float x = t.a.x - cx, y = t.a.y - cy, z = t.a.z - cz;
    const float d = t.u.x * x + t.u.y * y + t.u.z * z;
    // 1e-6, 1.0001: rounding of the normal, the difference and the two sums
    const float r = (fabsf(t.u.x) + fabsf(t.u.y) + fabsf(t.u.z)) * h * 1.0001f + 1e-6f * (fabsf(x) + fabsf(y) + fabsf(z));
    return !(fabsf(d) > r);
}

__device__ __forceinline__ int clamp_cell(float x, int n) {
    return x >= float(n) ? n - 1 : (x > 0.0f ? int(x) : 0);   // NaN: 0
}

// The coarse cells whose widened box a triangle's bounding box meets.
__device__ __forceinline__ bool cell_range(const Grid& g, const TriBox& t, int3& lo, int3& n) {
    const float inv = 1.0f / g.cell, r = g.reach + t.grow;
    if (t.hi.x < g.lox - r || t.lo.x > g.lox + g.nx * g.cell + r || t.hi.y < g.loy - r ||
        t.lo.y > g.loy + g.ny * g.cell + r || t.hi.z < g.loz - r || t.lo.z > g.loz + g.nz * g.cell + r)
        return false;
    // half a margin more on each side: the divisions' rounding
    const float e = r + 1e-3f * g.cell;
    lo = make_int3(clamp_cell((t.lo.x - e - g.lox) * inv, g.nx), clamp_cell((t.lo.y - e - g.loy) * inv, g.ny),
                   clamp_cell((t.lo.z - e - g.loz) * inv, g.nz));
    const int3 hi = make_int3(clamp_cell((t.hi.x + e - g.lox) * inv, g.nx), clamp_cell((t.hi.y + e - g.loy) * inv, g.ny),
                              clamp_cell((t.hi.z + e - g.loz) * inv, g.nz));
    n = make_int3(hi.x - lo.x + 1, hi.y - lo.y + 1, hi.z - lo.z + 1);
    return true;
}

__device__ __forceinline__ bool near_cell(const Grid& g, const TriBox& t, int x, int y, int z) {
    return near_box(t, g.lox + (x + 0.5f) * g.cell, g.loy + (y + 0.5f) * g.cell, g.loz + (z + 0.5f) * g.cell,
                    0.5f * g.cell + g.reach);
}

// Pass over the (triangle, coarse cell) pairs.  Count: count[cell] += 1.
// Fill: append the triangle to its cells' candidate lists.
struct Lists {
    uint32_t* count;            // per coarse cell (Count)
    const int32_t* top;         // per coarse cell: brick (Fill)
    const uint64_t* start;      // per brick: first entry of its list (Fill)
    uint32_t* cursor;           // per brick (Fill)
    int32_t* entry;             // candidate triangles (Fill)
};

template <bool kFill>
__device__ __forceinline__ void visit(const Grid& g, const Lists& l, int x, int y, int z, int t) {
    const size_t c = (size_t(z) * g.ny + y) * g.nx + x;
    if constexpr (kFill) {
        const int b = l.top[c];
        l.entry[l.start[b] + atomicAdd(l.cursor + b, 1u)] = t;
    } else {
        atomicAdd(l.count + c, 1u);
    }
}

// One warp per triangle; triangles over many cells are listed for big_kernel.
template <bool kFill>
__global__ void __launch_bounds__(256) small_kernel(const float4* tri, int n_tri, Grid g, Lists l, int32_t* big,
                                                    uint32_t* n_big) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < n_tri; t += warps) {
        const TriBox b = load_tri(tri, t, g);
        int3 lo, n;
        if (!cell_range(g, b, lo, n)) continue;
        const long long cells = (long long)n.x * n.y * n.z;
        if (cells > kBigCells) {
            if (!kFill && lane == 0) big[atomicAdd(n_big, 1u)] = t;
            continue;
        }
        for (int i = lane; i < int(cells); i += 32) {
            const int x = lo.x + i % n.x, y = lo.y + (i / n.x) % n.y, z = lo.z + i / (n.x * n.y);
            if (near_cell(g, b, x, y, z)) visit<kFill>(g, l, x, y, z, t);
        }
    }
}

template <bool kFill>
__global__ void __launch_bounds__(256) big_kernel(const float4* tri, Grid g, Lists l, const int32_t* big,
                                                  const uint32_t* n_big) {
    const uint32_t nb = *n_big;
    for (uint32_t k = 0; k < nb; ++k) {
        const int t = big[k];
        const TriBox b = load_tri(tri, t, g);
        int3 lo, n;
        if (!cell_range(g, b, lo, n)) continue;
        const long long cells = (long long)n.x * n.y * n.z;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cells;
             i += (long long)gridDim.x * blockDim.x) {
            const int x = lo.x + int(i % n.x), y = lo.y + int((i / n.x) % n.y), z = lo.z + int(i / ((long long)n.x * n.y));
            if (near_cell(g, b, x, y, z)) visit<kFill>(g, l, x, y, z, t);
        }
    }
}

// totals[0] += occupied cells, totals[1] += candidate entries
__global__ void __launch_bounds__(256) total_kernel(const uint32_t* count, uint64_t n, unsigned long long* totals) {
    unsigned long long c = 0, e = 0;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
        c += count[i] ? 1u : 0u;
        e += count[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if ((threadIdx.x & 31) == 0 && e) {
        atomicAdd(totals, c);
        atomicAdd(totals + 1, e);
    }
}

// Bricks of the occupied cells (numbered in arrival order); empty cells get
// kClearFar when their 26 neighbours are empty too, else kClearNear.
__global__ void __launch_bounds__(256) assign_kernel(const uint32_t* count, Grid g, unsigned long long* used,
                                                     int32_t* top, uint64_t* start, uint32_t* brick_cell) {
    const uint64_t n = uint64_t(g.nx) * g.ny * g.nz;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
        if (count[i]) {
            const uint32_t b = uint32_t(atomicAdd(used, 1ull));
            start[b] = atomicAdd(used + 1, (unsigned long long)count[i]);
            brick_cell[b] = uint32_t(i);
            top[i] = int(b);
            continue;
        }
        const int x = int(i % g.nx), y = int((i / g.nx) % g.ny), z = int(i / (uint64_t(g.nx) * g.ny));
        bool far = true;
        for (int dz = max(z - 1, 0); dz <= min(z + 1, g.nz - 1) && far; ++dz)
            for (int dy = max(y - 1, 0); dy <= min(y + 1, g.ny - 1) && far; ++dy)
                for (int dx = max(x - 1, 0); dx <= min(x + 1, g.nx - 1); ++dx)
                    if (count[(uint64_t(dz) * g.ny + dy) * g.nx + dx]) {
                        far = false;
                        break;
                    }
        top[i] = far ? dev::kClearFar : dev::kClearNear;
    }
}

// Extent along n of the part of a triangle inside the box of half edge h
// round the origin; false when there is none.  A triangle that lies in the
// box, or whose extent along n is next to nothing anyway (a flat face under
// its own normal), counts whole; the others are clipped (Sutherland-Hodgman,
// in local memory: on a flat geometry it was most of the map's time).
__device__ bool clipped_extent(float3 p0, float3 p1, float3 p2, float h, float3 n, float flat, float& lo, float& hi) {
    const float d0 = n.x * p0.x + n.y * p0.y + n.z * p0.z, d1 = n.x * p1.x + n.y * p1.y + n.z * p1.z,
                d2 = n.x * p2.x + n.y * p2.y + n.z * p2.z;
    lo = min3(d0, d1, d2);
    hi = max3(d0, d1, d2);
    const float reach = max3(max3(fabsf(p0.x), fabsf(p0.y), fabsf(p0.z)), max3(fabsf(p1.x), fabsf(p1.y), fabsf(p1.z)),
                             max3(fabsf(p2.x), fabsf(p2.y), fabsf(p2.z)));
    if (reach <= h || hi - lo <= flat) return true;
    // a convex polygon gains at most one vertex per plane (nine in all); one
    // that rounding has folded could gain more, and keeps what it has then
    // (clipping less only widens the extent)
    constexpr int kMax = 20;
    float3 v[kMax], w[kMax];
    v[0] = p0;
    v[1] = p1;
    v[2] = p2;
    int k = 3;
    for (int side = 0; side < 6 && k <= kMax / 2; ++side) {
        const int ax = side >> 1;
        const float s = (side & 1) ? -1.0f : 1.0f;
        int m = 0;
        for (int i = 0; i < k; ++i) {
            const float3 a = v[i], b = v[i + 1 < k ? i + 1 : 0];
            const float da = h - s * (ax == 0 ? a.x : ax == 1 ? a.y : a.z);
            const float db = h - s * (ax == 0 ? b.x : ax == 1 ? b.y : b.z);
            if (da >= 0.0f) w[m++] = a;
            if ((da >= 0.0f) != (db >= 0.0f)) {
                const float f = da / (da - db);
                w[m++] = make_float3(a.x + f * (b.x - a.x), a.y + f * (b.y - a.y), a.z + f * (b.z - a.z));
            }
        }
        k = m;
        if (k == 0) return false;
        for (int i = 0; i < k; ++i) v[i] = w[i];
    }
    lo = hi = n.x * v[0].x + n.y * v[0].y + n.z * v[0].z;
    for (int i = 1; i < k; ++i) {
        const float d = n.x * v[i].x + n.y * v[i].y + n.z * v[i].z;
        lo = fminf(lo, d);
        hi = fmaxf(hi, d);
    }
    return true;
}

// +1 / -1: u lies within 45 degrees of n / of -n; 0: neither
__device__ __forceinline__ float alike(float3 u, float3 n) {
    const float d = u.x * n.x + u.y * n.y + u.z * n.z;
    return d > 0.7f ? 1.0f : (d < -0.7f ? -1.0f : 0.0f);
}

// One block of 64 threads per brick, one thread per fine cell.  The first slab
// holds the candidates whose normals lie within 45 degrees of the nearest
// one's, the second the others; each slab's normal is the mean of its
// candidates' normals near that of its nearest, its extent that of its
// candidates' clipped parts, each widened by its margin.
__global__ void __launch_bounds__(kBrick * kBrick * kBrick) record_kernel(const float4* tri, Grid g, const uint32_t* brick_cell,
                                                                         const uint64_t* start, const uint32_t* n_entry,
                                                                         const int32_t* entry, float margin, float rounding,
                                                                         float4* rec) {
    const uint32_t b = blockIdx.x;
    const uint32_t c = brick_cell[b];
    const int cx = int(c % g.nx), cy = int((c / g.nx) % g.ny), cz = int(c / (uint32_t(g.nx) * g.ny));
    const int i = threadIdx.x;
    const float h = g.cell / kBrick;
    const float px = g.lox + (float(cx * kBrick + (i & 3)) + 0.5f) * h, py = g.loy + (float(cy * kBrick + ((i >> 2) & 3)) + 0.5f) * h,
                pz = g.loz + (float(cz * kBrick + (i >> 4)) + 0.5f) * h;
    const float box = 0.5f * h + g.reach;
    const int32_t* list = entry + start[b];
    const int n = int(n_entry[b]);
    float3 first = make_float3(0.0f, 0.0f, 0.0f);   // normal that marks the first slab's candidates
#pragma unroll 1
    for (int slab = 0; slab < 2; ++slab) {
        // this slab's nearest candidate
        float best = INFINITY;
        int bi = -1;
        float3 near = make_float3(0.0f, 0.0f, 0.0f);
        for (int k = 0; k < n; ++k) {
            const int t = __ldg(list + k);
            const TriBox tb = load_tri(tri, t, g);
            if (!near_box(tb, px, py, pz, box) || (slab == 1 && alike(tb.u, first) != 0.0f)) continue;
            const float d2 = dev::dist2_to_triangle(tri, t, px, py, pz);
            // (ties: the lowest index, so that the record does not depend on the list's order)
            if (d2 < best || (d2 == best && t < bi) || bi < 0) {
                best = d2;
                bi = t;
                near = tb.u;
            }
        }
        float4 out = make_float4(0.0f, 0.0f, 0.0f, -2.0f);   // nothing near: n . q - c = 2 everywhere
        // a first slab without a normal (zero area) takes every candidate
        const bool all = slab == 0 && bi >= 0 && near.x == 0.0f && near.y == 0.0f && near.z == 0.0f;
        if (bi >= 0) {
            if (slab == 0) first = near;
            float sx = 0.0f, sy = 0.0f, sz = 0.0f;
            for (int k = 0; k < n; ++k) {
                const TriBox tb = load_tri(tri, __ldg(list + k), g);
                if (!near_box(tb, px, py, pz, box)) continue;
                if (slab == 1 && alike(tb.u, first) != 0.0f) continue;
                const float s = alike(tb.u, near);
                sx += s * tb.u.x;
                sy += s * tb.u.y;
                sz += s * tb.u.z;
            }
            float l2 = sx * sx + sy * sy + sz * sz;
            if (!(l2 > 1e-12f)) {   // no usable normal (degenerate triangles): any direction serves
                sx = sy = 0.0f;
                sz = l2 = 1.0f;
            }
            const float s = rsqrtf(l2);
            const float3 u = make_float3(sx * s, sy * s, sz * s);
            float lo = INFINITY, hi = -INFINITY;
            for (int k = 0; k < n; ++k) {
                const TriBox tb = load_tri(tri, __ldg(list + k), g);
                if (!near_box(tb, px, py, pz, box)) continue;
                if (!all && (alike(tb.u, first) != 0.0f) != (slab == 0)) continue;
                const float3 p0 = make_float3(tb.a.x - px, tb.a.y - py, tb.a.z - pz);
                const float co = tb.u.x * u.x + tb.u.y * u.y + tb.u.z * u.z;
                const float m = fmaxf(margin, tb.slack * (0.5f + 10.0f * sqrtf(fmaxf(1.0f - co * co, 0.0f)))) + rounding;
                float a, e;
                if (clipped_extent(p0, make_float3(p0.x + tb.e1.x, p0.y + tb.e1.y, p0.z + tb.e1.z),
                                   make_float3(p0.x + tb.e2.x, p0.y + tb.e2.y, p0.z + tb.e2.z), box + tb.grow, u,
                                   0.1f * margin, a, e)) {
                    lo = fminf(lo, a - m);
                    hi = fmaxf(hi, e + m);
                }
            }
            if (hi - lo < 1e6f * g.reach) {
                const float inv = 2.0f / (hi - lo);
                out = make_float4(u.x * inv, u.y * inv, u.z * inv, 0.5f * (hi + lo) * inv);
            } else if (hi >= lo) {
                out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   // no bound on a candidate's rounding: every step walks
            }
        }
        rec[2 * (size_t(b) * (kBrick * kBrick * kBrick) + i) + slab] = out;
        if (all) {   // nothing is left for the second slab
            rec[2 * (size_t(b) * (kBrick * kBrick * kBrick) + i) + 1] = make_float4(0.0f, 0.0f, 0.0f, -2.0f);
            return;
        }
    }
}

// One device allocation cut into arrays: allocating and freeing cost more
// than the map's kernels on small geometries.
struct Block {
    unsigned char* p = nullptr;
    size_t used = 0;
    ~Block() {
        if (p) cudaFree(p);
    }
    // Reserves n elements; their address is valid after alloc.
    template <typename T>
    size_t reserve(uint64_t n) {
        const size_t at = used;
        used += (std::max<uint64_t>(n, 1) * sizeof(T) + 255) / 256 * 256;
        return at;
    }
    bool alloc() {
        if (cudaMalloc(&p, used) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return p != nullptr;
    }
    template <typename T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(p + offset);
    }
};

}  // namespace

// Cell size: kFineCell, doubled until the coarse grid and the records fit
// their budgets (kMaxCells coarse cells; an eighth of the free memory, at
// most kMaxRecordBytes, for the records).  The reach grows with the cells.
bool build_clearance(const float4* tri, int n_tri, const float center[3], const float half[3], int sms, cudaStream_t s,
                     ClearanceMap* out) {
    constexpr float kFineCell = 4.0f, kReach = 3.0f;
    constexpr uint64_t kMaxCells = 1ull << 26, kMaxRecordBytes = 4ull << 30;
    constexpr uint64_t kBrickCells = kBrick * kBrick * kBrick, kRecordBytes = 2 * sizeof(float4);
    float scale = 0.0f;   // largest coordinate: sizes the rounding margin
    for (int i = 0; i < 3; ++i) {
        if (!(half[i] > 0.0f) || !(half[i] < 1e18f) || !(std::fabs(center[i]) < 1e18f)) return false;
        scale = std::max(scale, std::fabs(center[i]) + half[i]);
    }
    size_t free_b = 0, total_b = 0;
    if (n_tri <= 0 || cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const uint64_t budget = std::min<uint64_t>(free_b / 8, kMaxRecordBytes);
    // Rounding: positions, the records and the transport's own test are single
    // precision at magnitudes up to `scale` (half an ulp: 6e-8 scale); 4e-6
    // leaves a factor of sixty.  0.02 nm on top keeps steps that graze a
    // triangle's edge on the exact path (0.05 nm: contact holes, whose
    // electrons hug the interfaces, 28.9 instead of 26.8 ms).
    const float margin = 0.02f, rounding = 4e-6f * scale;
    const int blocks = sms * 8;
    float fine = kFineCell, reach = kReach;
    for (int tries = 0; tries < 24; ++tries, fine *= 2.0f, reach *= 2.0f) {
        Grid g{};
        g.cell = fine * kBrick;
        g.reach = reach + margin + rounding;
        g.lox = center[0] - half[0];
        g.loy = center[1] - half[1];
        g.loz = center[2] - half[2];
        double dims[3];
        for (int i = 0; i < 3; ++i) dims[i] = std::ceil(2.0 * double(half[i]) / double(g.cell)) + 1.0;
        // (below 2^22 fine cells an axis: the transport's index arithmetic)
        if (dims[0] * dims[1] * dims[2] > double(kMaxCells) || std::max({dims[0], dims[1], dims[2]}) > double(1 << 19))
            continue;
        g.nx = int(dims[0]);
        g.ny = int(dims[1]);
        g.nz = int(dims[2]);
        const uint64_t cells = uint64_t(g.nx) * g.ny * g.nz;
        // counting pass: the first words and the counts start at zero
        Block first;
        const size_t at_totals = first.reserve<unsigned long long>(4), at_n_big = first.reserve<uint32_t>(1),
                     at_count = first.reserve<uint32_t>(cells), zeroed = first.used,
                     at_big = first.reserve<int32_t>(uint64_t(n_tri));
        if (!first.alloc() || cudaMemsetAsync(first.p, 0, zeroed, s) != cudaSuccess) return false;
        unsigned long long* const totals = first.at<unsigned long long>(at_totals);
        uint32_t *const n_big = first.at<uint32_t>(at_n_big), *const count = first.at<uint32_t>(at_count);
        int32_t* const big = first.at<int32_t>(at_big);
        Lists l{};
        l.count = count;
        small_kernel<false><<<blocks, 256, 0, s>>>(tri, n_tri, g, l, big, n_big);
        big_kernel<false><<<blocks, 256, 0, s>>>(tri, g, l, big, n_big);
        total_kernel<<<blocks, 256, 0, s>>>(count, cells, totals);
        unsigned long long used[2] = {0, 0};
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(used, totals, 16, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return false;
        if (used[0] * kBrickCells * kRecordBytes > budget || used[1] * 4 > budget) continue;
        Block lists, map;
        const size_t at_entry = lists.reserve<int32_t>(used[1]), at_start = lists.reserve<uint64_t>(used[0]),
                     at_cell = lists.reserve<uint32_t>(used[0]), at_cursor = lists.reserve<uint32_t>(used[0]);
        const size_t at_rec = map.reserve<float4>(std::max<uint64_t>(used[0], 1) * kBrickCells * 2),
                     at_top = map.reserve<int32_t>(cells);
        if (!lists.alloc() || !map.alloc()) return false;
        uint32_t *const brick_cell = lists.at<uint32_t>(at_cell), *const cursor = lists.at<uint32_t>(at_cursor);
        uint64_t* const start = lists.at<uint64_t>(at_start);
        int32_t* const top = map.at<int32_t>(at_top);
        float4* const rec = map.at<float4>(at_rec);
        if (cudaMemsetAsync(cursor, 0, 4 * std::max<uint64_t>(used[0], 1), s) != cudaSuccess) return false;
        assign_kernel<<<blocks, 256, 0, s>>>(count, g, totals + 2, top, start, brick_cell);
        l.top = top;
        l.start = start;
        l.cursor = cursor;
        l.entry = lists.at<int32_t>(at_entry);
        small_kernel<true><<<blocks, 256, 0, s>>>(tri, n_tri, g, l, big, n_big);
        big_kernel<true><<<blocks, 256, 0, s>>>(tri, g, l, big, n_big);
        if (used[0])
            record_kernel<<<unsigned(used[0]), unsigned(kBrickCells), 0, s>>>(tri, g, brick_cell, start, cursor, l.entry,
                                                                              margin, rounding, rec);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return false;
        out->memory = map.p;
        map.p = nullptr;
        dev::Clearance& m = out->map;
        m.top = top;
        m.rec = rec;
        m.offx = float(-double(g.lox) / fine - 0.5);
        m.offy = float(-double(g.loy) / fine - 0.5);
        m.offz = float(-double(g.loz) / fine - 0.5);
        m.midx = g.lox + 0.5f * fine;
        m.midy = g.loy + 0.5f * fine;
        m.midz = g.loz + 0.5f * fine;
        m.h = fine;
        m.inv_h = 1.0f / fine;
        m.nx = g.nx;
        m.ny = g.ny;
        m.reach = reach;
        m.far_reach = g.cell;
        return true;
    }
    return false;
}

void free_clearance(ClearanceMap* m) {
    if (m->memory) cudaFree(m->memory);
    *m = ClearanceMap{};
}

}  // namespace nbx
