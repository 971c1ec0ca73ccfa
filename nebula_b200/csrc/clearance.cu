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
// triangle" has to mean that intersect_ray reports no hit.  With u = 2^-24, s
// the vector from the triangle's corner to the ray's start and k = |e1||e2| /
// |e1 x e2|, the test's numerators u and v are off by at most 12 u |s| times the
// edge in them, its determinant by 8 u |e1||e2| and the numerator of t by
// 6 u |e2| . (|s| x |e1|), the triple product of the vectors' magnitudes by
// component with its differences taken as sums.  So the point that it reports
// lies
// * along the triangle's normal within that triple product's 6 u / |e1 x e2|
//   (small where the plane runs along an axis, 12 u k |s| at most) and 8 u k
//   times the step,
// * in the triangle's plane within 44 u k |s| / cos of it, cos being that of the
//   ray's angle to the normal, and the 2.4e-6 of the edges by which the test
//   enlarges a triangle.
// A triangle at an angle phi to its slab widens the slab by the first and by the
// second times sin(phi), with 240 u in place of 44 u / cos: rays down to a cosine
// of 0.18 at the bound and of 0.02 at the errors that occur (a tenth of it).  It
// is a candidate of the cells that its plane meets within the first bound and
// that lie within the second of it.  On the benchmark scans all this is below
// 0.01 nm for most triangles, and the margin decides; strips of 1000 nm x 0.3 nm
// at an angle to one another make the cells round them walk.  With one margin for
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

struct alignas(16) TriBox {
    float3 a, e1, e2, lo, hi;
    float3 u;      // unit normal (zero without an area)
    float k;       // |e1||e2| / |e1 x e2| (infinite without an area)
    float inv;     // 1 / |e1 x e2|
    float size;    // diagonal of the bounding box
    float thick;   // rounding of the exact test along the normal, at most (nm)
    float grow;    // and in the plane (nm)
};

__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(a, fminf(b, c)); }
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(a, fmaxf(b, c)); }

constexpr float kUnit = 5.9604645e-8f;         // 2^-24
constexpr float kReachDiagonal = 1.7320508f;   // of a cube of edge 1

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
    r.k = s > 0.0 ? sqrtf(b2) * sqrtf(c2) * float(s) : INFINITY;
    r.inv = s > 0.0 ? float(s) : INFINITY;
    const float dx = r.hi.x - r.lo.x, dy = r.hi.y - r.lo.y, dz = r.hi.z - r.lo.z;
    r.size = sqrtf(dx * dx + dy * dy + dz * dz);   // at least the longest edge
    // |s| of rays in a widened fine cell near the triangle (kReachDiagonal: its diagonal)
    const float far = 1.25f * r.size + kReachDiagonal * (g.cell / kBrick + 2.0f * g.reach);
    r.thick = 20.0f * kUnit * r.k * far;
    // (capped: a hit farther off than twice the triangle's size takes a ray whose
    // line meets it to one part in 1e7 and a distance that is all rounding)
    r.grow = fminf(240.0f * kUnit * r.k * far + 2.4e-6f * r.size, fminf(2.0f * r.size, 8.0f * g.cell));
    // The exact test drops a triangle whose determinant is below kEps, rounding
    // included, for every ray: it is near nothing (exported meshes hold many
    // such triangles, of no area and short edges, on their surfaces).
    if (l2 < 1e-10 && sqrtf(float(l2)) + 10.0f * kUnit * sqrtf(b2) * sqrtf(c2) < 0.99f * dev::kEps)
        r.lo = make_float3(INFINITY, INFINITY, INFINITY);
    return r;
}

// Conservative triangle / box test: bounding boxes, then the triangle's
// plane against the box.  (cx, cy, cz) is the box centre, h its half edge.
__device__ __forceinline__ bool near_box(const TriBox& t, float cx, float cy, float cz, float h) {
    const float w = h + t.grow;
    if (t.lo.x > cx + w || t.hi.x < cx - w || t.lo.y > cy + w || t.hi.y < cy - w || t.lo.z > cz + w || t.hi.z < cz - w)
        return false;
    const float x = t.a.x - cx, y = t.a.y - cy, z = t.a.z - cz;
    const float d = t.u.x * x + t.u.y * y + t.u.z * z;
    // 1e-6, 1.0001: rounding of the normal, the difference and the two sums
    const float r = (fabsf(t.u.x) + fabsf(t.u.y) + fabsf(t.u.z)) * h * 1.0001f + 1e-6f * (fabsf(x) + fabsf(y) + fabsf(z));
    return !(fabsf(d) > r + t.thick);
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
// round the origin; false when there is none.  p is the triangle's corner.  A
// triangle that lies in the box, or whose extent along n is next to nothing
// anyway (a flat face under its own normal), counts whole.  For the others the
// part's corners are the ends of the triangle's edges inside the box and the
// points where the box's edges pass through the triangle.  (A corner that
// rounding loses lies within it of one that is kept.)  No polygon is kept:
// clipping plane by plane needs arrays in local memory, which were most of the
// map's time.
__device__ __forceinline__ bool clipped_extent(const TriBox& t, float3 p, float h, float3 n, float flat, float& lo, float& hi) {
    const float3 e1 = t.e1, e2 = t.e2;
    const float dp = n.x * p.x + n.y * p.y + n.z * p.z, d1 = n.x * e1.x + n.y * e1.y + n.z * e1.z,
                d2 = n.x * e2.x + n.y * e2.y + n.z * e2.z;
    lo = dp + min3(0.0f, d1, d2);
    hi = dp + max3(0.0f, d1, d2);
    const float far = max3(max3(fabsf(p.x), fabsf(p.y), fabsf(p.z)),
                           max3(fabsf(p.x + e1.x), fabsf(p.y + e1.y), fabsf(p.z + e1.z)),
                           max3(fabsf(p.x + e2.x), fabsf(p.y + e2.y), fabsf(p.z + e2.z)));
    if (far <= h || hi - lo <= flat) return true;
    lo = INFINITY;
    hi = -INFINITY;
    // the triangle's edges: from a along d, in the box for parameters [s, e]
    auto edge = [&](float3 a, float3 d, float da, float dd) {
        const float ix = 1.0f / d.x, iy = 1.0f / d.y, iz = 1.0f / d.z;
        const float x0 = (-h - a.x) * ix, x1 = (h - a.x) * ix, y0 = (-h - a.y) * iy, y1 = (h - a.y) * iy,
                    z0 = (-h - a.z) * iz, z1 = (h - a.z) * iz;
        const float s = fmaxf(0.0f, max3(fminf(x0, x1), fminf(y0, y1), fminf(z0, z1)));
        const float e = fminf(1.0f, min3(fmaxf(x0, x1), fmaxf(y0, y1), fmaxf(z0, z1)));
        if (s <= e) {
            const float u = da + dd * s, v = da + dd * e;
            lo = min3(lo, u, v);
            hi = max3(hi, u, v);
        }
    };
    edge(p, e1, dp, d1);
    edge(p, e2, dp, d2);
    edge(make_float3(p.x + e1.x, p.y + e1.y, p.z + e1.z), make_float3(e2.x - e1.x, e2.y - e1.y, e2.z - e1.z), dp + d1, d2 - d1);
    // the box's edges along x, y and z: the point of the triangle's plane on
    // each, and its barycentric coordinates times twice the area, f, g and
    // area - f - g
    const float3 u = t.u, f1 = make_float3(u.y * e1.z - u.z * e1.y, u.z * e1.x - u.x * e1.z, u.x * e1.y - u.y * e1.x),
                 f2 = make_float3(u.y * e2.z - u.z * e2.y, u.z * e2.x - u.x * e2.z, u.x * e2.y - u.y * e2.x);
    const float area = f1.x * e2.x + f1.y * e2.y + f1.z * e2.z, at = u.x * p.x + u.y * p.y + u.z * p.z;
    const float size = fabsf(e1.x) + fabsf(e1.y) + fabsf(e1.z) + fabsf(e2.x) + fabsf(e2.y) + fabsf(e2.z);
    const float tol = -2e-6f * size * (size + 2.0f * h);
    auto corner = [&](float x, float y, float z) {
        const float rx = x - p.x, ry = y - p.y, rz = z - p.z;
        const float f = f1.x * rx + f1.y * ry + f1.z * rz, g = -(f2.x * rx + f2.y * ry + f2.z * rz);
        if (f >= tol && g >= tol && area - f - g >= tol) {
            const float d = n.x * x + n.y * y + n.z * z;
            lo = fminf(lo, d);
            hi = fmaxf(hi, d);
        }
    };
    const float ux = 1.0f / u.x, uy = 1.0f / u.y, uz = 1.0f / u.z;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float a = (k & 1) ? h : -h, b = (k & 2) ? h : -h;
        const float x = (at - u.y * a - u.z * b) * ux, y = (at - u.x * a - u.z * b) * uy, z = (at - u.x * a - u.y * b) * uz;
        if (fabsf(x) <= h) corner(x, a, b);
        if (fabsf(y) <= h) corner(a, y, b);
        if (fabsf(z) <= h) corner(a, b, z);
    }
    return hi >= lo;
}

// +1 / -1: u lies within 45 degrees of n / of -n; 0: neither
__device__ __forceinline__ float alike(float3 u, float3 n) {
    const float d = u.x * n.x + u.y * n.y + u.z * n.z;
    return d > 0.7f ? 1.0f : (d < -0.7f ? -1.0f : 0.0f);
}

// A slab of a fine cell while its record is made.
struct Slab {
    float best = INFINITY;   // nearest candidate: squared distance, index, normal
    int t = -1;
    float3 near = {0.0f, 0.0f, 0.0f};
    float3 sum = {0.0f, 0.0f, 0.0f};   // of the normals near that one
    float3 u = {0.0f, 0.0f, 1.0f};     // the slab's normal
    float lo = INFINITY, hi = -INFINITY;

    // (ties: the lowest index, so that the record does not depend on the list's order)
    __device__ __forceinline__ void nearest(const TriBox& b, int i, float px, float py, float pz) {
        float qx, qy, qz;
        dev::closest_point_on_triangle(px, py, pz, make_float4(b.a.x, b.a.y, b.a.z, 0.0f),
                                       make_float4(b.e1.x, b.e1.y, b.e1.z, 0.0f),
                                       make_float4(b.e2.x, b.e2.y, b.e2.z, 0.0f), &qx, &qy, &qz);
        const float d2 = (px - qx) * (px - qx) + (py - qy) * (py - qy) + (pz - qz) * (pz - qz);
        if (d2 < best || (d2 == best && i < t) || t < 0) {
            best = d2;
            t = i;
            near = b.u;
        }
    }
    __device__ __forceinline__ void add_normal(const TriBox& b) {
        const float s = alike(b.u, near);
        sum.x += s * b.u.x;
        sum.y += s * b.u.y;
        sum.z += s * b.u.z;
    }
    __device__ __forceinline__ void set_normal() {
        const float l2 = sum.x * sum.x + sum.y * sum.y + sum.z * sum.z;
        if (!(l2 > 1e-12f)) return;   // no usable normal (degenerate triangles): any direction serves
        const float s = rsqrtf(l2);
        u = make_float3(sum.x * s, sum.y * s, sum.z * s);
    }
    __device__ __forceinline__ void extend(const TriBox& b, float px, float py, float pz, float box, float margin,
                                           float rounding) {
        const float3 p = make_float3(b.a.x - px, b.a.y - py, b.a.z - pz);
        const float co = b.u.x * u.x + b.u.y * u.y + b.u.z * u.z;
        // magnitudes of s by component and in length, for rays that start in the box
        const float sx = fabsf(p.x) + box, sy = fabsf(p.y) + box, sz = fabsf(p.z) + box;
        const float ex = fabsf(b.e1.x), ey = fabsf(b.e1.y), ez = fabsf(b.e1.z);
        const float triple = fabsf(b.e2.x) * (sy * ez + sz * ey) + fabsf(b.e2.y) * (sz * ex + sx * ez) +
                             fabsf(b.e2.z) * (sx * ey + sy * ex);
        const float along = kUnit * (6.0f * triple * b.inv + 8.0f * b.k * kReachDiagonal * box);
        const float across = 240.0f * kUnit * b.k * sqrtf(sx * sx + sy * sy + sz * sz) + 2.4e-6f * b.size;
        // (k is infinite without an area: no bound)
        const float si = sqrtf(fmaxf(1.0f - co * co, 0.0f)) + 5e-4f;   // (rounding of co near 1)
        const float m = b.k < 1e30f ? fmaxf(margin, along + across * si) + rounding : INFINITY;
        float x, y;
        if (clipped_extent(b, p, box + b.grow, u, 0.1f * margin, x, y)) {
            lo = fminf(lo, x - m);
            hi = fmaxf(hi, y + m);
        }
    }
    __device__ __forceinline__ float4 record(float most) const {
        if (!(hi >= lo)) return make_float4(0.0f, 0.0f, 0.0f, -2.0f);   // nothing near: n . q - c = 2 everywhere
        // no bound on a candidate's rounding: every step walks
        if (!(hi - lo < most)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float inv = 2.0f / (hi - lo);
        return make_float4(u.x * inv, u.y * inv, u.z * inv, 0.5f * (hi + lo) * inv);
    }
};

// One block of 64 threads per brick, one thread per fine cell.  The first slab
// holds the candidates whose normals lie within 45 degrees of the nearest
// one's, the second the others; each slab's normal is the mean of its
// candidates' normals near that of its nearest, its extent that of its
// candidates' clipped parts, each widened by its margin.
//
// Bound by the instructions of clipped_extent and near_box (a brick of the
// contact holes has 31 candidates).  The block keeps its candidates in shared
// memory, 64 at a time, and goes over them four times (nearest; normal, and the
// second slab's nearest; extent, and the second slab's normal; the second slab's
// extent).  B200, against every thread reading
// and preparing every candidate six times and clipping polygons in local
// memory: 16 x 16 contact holes (89,067 bricks, 2.8 million candidates) 16.2 ->
// 6.7 ms, 8 x 8 holes 4.5 -> 1.8 ms; nbx_set_geometry 29 -> 21 and 9.0 -> 6.9 ms,
// of which 11 and 3 ms are the octree and the triangles.
//
// A brick of more than kMaxList candidates (a mesh far finer than the cells, as
// in a domain that is far larger) gets records under which every step walks:
// there its slabs would fill their cells, and finding that out took 370 ms for
// 132,108 triangles in one cell of a 1 mm domain (8 ms with the limit).
constexpr int kMaxList = 1 << 14;
__global__ void __launch_bounds__(kBrick * kBrick * kBrick) record_kernel(const float4* tri, Grid g, const uint32_t* brick_cell,
                                                                         const uint64_t* start, const uint32_t* n_entry,
                                                                         const int32_t* entry, float margin, float rounding,
                                                                         float4* rec) {
    constexpr int kTile = kBrick * kBrick * kBrick;
    __shared__ TriBox tile[kTile];
    __shared__ int tile_t[kTile];
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
    float4* const out = rec + 2 * (size_t(b) * kTile + i);
    if (n > kMaxList) {   // (the whole block)
        out[0] = out[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    bool loaded = false;
    // f(candidate, index) for the candidates near this thread's cell; called by the whole block
    auto each = [&](auto&& f) {
        for (int at = 0; at < n; at += kTile) {
            if (!loaded || n > kTile) {
                __syncthreads();
                if (at + i < n) {
                    tile_t[i] = __ldg(list + at + i);
                    tile[i] = load_tri(tri, tile_t[i], g);
                }
                __syncthreads();
                loaded = true;
            }
            const int m = min(kTile, n - at);
            for (int k = 0; k < m; ++k)
                if (near_box(tile[k], px, py, pz, box)) f(tile[k], tile_t[k]);
        }
    };
    Slab s0, s1;
    each([&](const TriBox& t, int k) { s0.nearest(t, k, px, py, pz); });
    // (a first slab without a normal, of a triangle without an area, takes every candidate)
    const bool all = s0.near.x == 0.0f && s0.near.y == 0.0f && s0.near.z == 0.0f;
    auto in_first = [&](const TriBox& t) { return all || alike(t.u, s0.near) != 0.0f; };
    each([&](const TriBox& t, int k) {
        if (in_first(t))
            s0.add_normal(t);
        else
            s1.nearest(t, k, px, py, pz);
    });
    s0.set_normal();
    each([&](const TriBox& t, int) {
        if (in_first(t))
            s0.extend(t, px, py, pz, box, margin, rounding);
        else
            s1.add_normal(t);
    });
    if (__syncthreads_or(s1.t >= 0)) {
        s1.set_normal();
        each([&](const TriBox& t, int) {
            if (!in_first(t)) s1.extend(t, px, py, pz, box, margin, rounding);
        });
    }
    out[0] = s0.record(1e6f * g.reach);
    out[1] = s1.record(1e6f * g.reach);
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
    cudaError_t alloc() {
        const cudaError_t e = cudaMalloc(&p, used);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return e;
    }
    template <typename T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(p + offset);
    }
};

}  // namespace

// Cell size: kFineCell, doubled until the map, and the lists it is made from,
// each fit an eighth of the free memory (at most kMaxBytes) and can be
// allocated, with at most kMaxCells coarse cells.  The reach grows with the
// cells.
cudaError_t build_clearance(const float4* tri, int n_tri, const float center[3], const float half[3], int sms,
                            cudaStream_t s, ClearanceMap* out) {
    constexpr float kFineCell = 4.0f, kReach = 3.0f;
    constexpr uint64_t kMaxCells = 1ull << 26, kMaxBytes = 4ull << 30;
    constexpr uint64_t kBrickCells = kBrick * kBrick * kBrick;
    float scale = 0.0f;   // largest coordinate: sizes the rounding margin
    for (int i = 0; i < 3; ++i) {
        if (!(half[i] > 0.0f) || !(half[i] < 1e18f) || !(std::fabs(center[i]) < 1e18f)) return cudaSuccess;
        scale = std::max(scale, std::fabs(center[i]) + half[i]);
    }
    if (n_tri <= 0) return cudaSuccess;
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    const uint64_t budget = std::min<uint64_t>(free_b / 8, kMaxBytes);
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
        if (cells * sizeof(int32_t) > budget) continue;
        // counting pass: the first words and the counts start at zero
        Block first;
        const size_t at_totals = first.reserve<unsigned long long>(4), at_n_big = first.reserve<uint32_t>(1),
                     at_count = first.reserve<uint32_t>(cells), zeroed = first.used,
                     at_big = first.reserve<int32_t>(uint64_t(n_tri));
        e = first.alloc();
        if (e == cudaErrorMemoryAllocation) continue;
        if (e != cudaSuccess || (e = cudaMemsetAsync(first.p, 0, zeroed, s)) != cudaSuccess) return e;
        unsigned long long* const totals = first.at<unsigned long long>(at_totals);
        uint32_t *const n_big = first.at<uint32_t>(at_n_big), *const count = first.at<uint32_t>(at_count);
        int32_t* const big = first.at<int32_t>(at_big);
        Lists l{};
        l.count = count;
        small_kernel<false><<<blocks, 256, 0, s>>>(tri, n_tri, g, l, big, n_big);
        big_kernel<false><<<blocks, 256, 0, s>>>(tri, g, l, big, n_big);
        total_kernel<<<blocks, 256, 0, s>>>(count, cells, totals);
        unsigned long long used[2] = {0, 0};
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = cudaMemcpyAsync(used, totals, 16, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        Block lists, map;
        const size_t at_entry = lists.reserve<int32_t>(used[1]), at_start = lists.reserve<uint64_t>(used[0]),
                     at_cell = lists.reserve<uint32_t>(used[0]), at_cursor = lists.reserve<uint32_t>(used[0]);
        const size_t at_rec = map.reserve<float4>(std::max<uint64_t>(used[0], 1) * kBrickCells * 2),
                     at_top = map.reserve<int32_t>(cells);
        if (map.used > budget || lists.used > budget) continue;
        e = lists.alloc();
        if (e == cudaSuccess) e = map.alloc();
        if (e == cudaErrorMemoryAllocation) continue;
        if (e != cudaSuccess) return e;
        uint32_t *const brick_cell = lists.at<uint32_t>(at_cell), *const cursor = lists.at<uint32_t>(at_cursor);
        uint64_t* const start = lists.at<uint64_t>(at_start);
        int32_t* const top = map.at<int32_t>(at_top);
        float4* const rec = map.at<float4>(at_rec);
        if ((e = cudaMemsetAsync(cursor, 0, 4 * std::max<uint64_t>(used[0], 1), s)) != cudaSuccess) return e;
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
        if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
        out->memory = map.p;
        out->bytes = map.used;
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
        return cudaSuccess;
    }
    return cudaSuccess;
}

void free_clearance(ClearanceMap* m) {
    if (m->memory) cudaFree(m->memory);
    *m = ClearanceMap{};
}

}  // namespace nbx
