// Electrode surfaces: a triangle mesh that stops particles whose step segment
// crosses it.
//
// Reference: Pusher.track_batch tests each step's segment (position before
// -> after the push) of every active particle against the electrode assembly
// and deactivates the ones that hit (src/PyPATools/pusher.py:970-990, calling
// PyElectrodeAssembly.segment_intersects_surface of the external py_electrodes
// package).  Here the surface is a triangle mesh on the device, binned into a
// uniform grid of cells; a segment is tested against the triangles of the
// cells its bounding box overlaps with the Moller-Trumbore ray-triangle test
// (T. Moller, B. Trumbore, "Fast, minimum storage ray-triangle
// intersection", J. Graphics Tools 2(1), 1997), restricted to the segment
// (0 <= t <= 1, edges and end points included).
//
// The test's arithmetic is written with explicitly rounded operations (no
// fused multiply-adds) in a fixed order, so every hit decision is the same
// as the NumPy restatement's, bit for bit.
#pragma once

#include <mutex>
#include <vector>

#include "ppt_internal.cuh"

namespace ppt {

struct SurfaceDev {
    const double* tri;          // 9 per triangle: v0, e1 = v1 - v0, e2 = v2 - v0
    const int32_t* cell_start;  // cells + 1 offsets into cell_tri
    const int32_t* cell_tri;    // triangle indices, binned by cell ([i][j][k], k fastest)
    double lo[3];               // grid origin
    double inv_h[3];            // 1 / cell size
    int32_t dims[3];
    int32_t n_tri;
    const int32_t* trange;      // 6 per triangle: its first and last cell per axis (x0 x1 y0 y1 z0 z1)
    // the grid the segment test uses: every cell cut into a few per axis
    // (ppt_surface_refine; before it, the cells themselves)
    const int32_t* seg_start;
    const int32_t* seg_tri;
    double seg_h[3];
    double seg_inv_h[3];
    int32_t seg_dims[3];
    const double* plane;        // 4 per triangle: its plane's normal and offset (see beyond_plane)
    double centre[3];           // the point the planes' offsets are from
    double reach;               // the farthest the grid goes from it
    const uint8_t* clearance;   // per cell: how many cells away (along any axis) the nearest listed triangle is,
                                // at most 255 (NULL before ppt_surface_refine: no clear boxes)
    double h[3];                // cell size
};

__device__ __forceinline__ double rn_dot(double ax, double ay, double az, double bx, double by, double bz) {
    return __dadd_rn(__dadd_rn(__dmul_rn(ax, bx), __dmul_rn(ay, by)), __dmul_rn(az, bz));
}

__device__ __forceinline__ V3 rn_cross(V3 a, V3 b) {
    return v3(__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(a.z, b.y)),
              __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(a.x, b.z)),
              __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}

// Segment p0 + t d, t in [0, 1], against one triangle.
__device__ __forceinline__ bool segment_hits_triangle(const double* __restrict__ T, V3 p0, V3 d) {
    const V3 v0 = v3(T[0], T[1], T[2]);
    const V3 e1 = v3(T[3], T[4], T[5]);
    const V3 e2 = v3(T[6], T[7], T[8]);
    const V3 pv = rn_cross(d, e2);
    const double det = rn_dot(e1.x, e1.y, e1.z, pv.x, pv.y, pv.z);
    if (det == 0.0) return false;   // the segment is parallel to the triangle's plane
    const double inv = 1.0 / det;
    const V3 tv = v3(__dsub_rn(p0.x, v0.x), __dsub_rn(p0.y, v0.y), __dsub_rn(p0.z, v0.z));
    const double u = __dmul_rn(rn_dot(tv.x, tv.y, tv.z, pv.x, pv.y, pv.z), inv);
    if (!(u >= 0.0 && u <= 1.0)) return false;
    const V3 qv = rn_cross(tv, e1);
    const double v = __dmul_rn(rn_dot(d.x, d.y, d.z, qv.x, qv.y, qv.z), inv);
    if (!(v >= 0.0 && __dadd_rn(u, v) <= 1.0)) return false;
    const double t = __dmul_rn(rn_dot(e2.x, e2.y, e2.z, qv.x, qv.y, qv.z), inv);
    return t >= 0.0 && t <= 1.0;
}

// Do both ends of a segment (a, b: from the planes' centre) lie on one side of
// a triangle's plane, farther from it than the rounding of segment_hits_triangle
// could bridge?  Then that test finds no hit.  With N = e1 x e2 it finds t as
// N.(p0 - v0) / N.(p0 - p1), each rounded to within a few 2^-53 |e1| |e2| L, L the
// lengths that enter; the planes are scaled by 1 / (|e1| |e2|), so a distance
// above `margin` = 2^-43 L decides as the test would.  Four numbers and six FMAs
// against nine and some fifty operations with a division: near a wall a step's
// cell lists ten triangles, nearly all of them away from the segment.
__device__ __forceinline__ bool beyond_plane(const double* __restrict__ plane, V3 a, V3 b, double margin) {
    double nx, ny, nz, w;
    ldg_f64x4(plane, nx, ny, nz, w);
    const double sa = fma(nx, a.x, fma(ny, a.y, fma(nz, a.z, w)));
    const double sb = fma(nx, b.x, fma(ny, b.y, fma(nz, b.z, w)));
    return (sa > margin && sb > margin) || (sa < -margin && sb < -margin);
}

// Any triangle listed by the cells lo .. hi of one of the grids.
__device__ __forceinline__ bool cells_hit(const SurfaceDev& S, const int32_t* __restrict__ start,
                                          const int32_t* __restrict__ list, int ny, int nz, const int lo[3],
                                          const int hi[3], V3 p0, V3 d, V3 from, V3 to, double margin) {
    for (int i = lo[0]; i <= hi[0]; ++i)
        for (int j = lo[1]; j <= hi[1]; ++j)
            for (int k = lo[2]; k <= hi[2]; ++k) {
                const int cell = (i * ny + j) * nz + k;
                const int end = start[cell + 1];
                for (int q = start[cell]; q < end; ++q) {
                    const int64_t tri = list[q];
                    if (beyond_plane(S.plane + 4 * tri, from, to, margin)) continue;
                    if (segment_hits_triangle(S.tri + 9 * tri, p0, d)) return true;
                }
            }
    return false;
}

// Does the segment p0 -> p1 meet any triangle of the surface?  The cells of
// the segment's bounding box are visited (one for the short steps of a
// tracking run); a triangle listed in several of them may be tested twice.
// A box of more than kSegMostVisits of the segment grid's cells takes the cells
// that were cut into them, up to 64 times fewer: a long segment visits many cells
// that list nothing, or the same triangles again.  2e5 segments beside a plate and a
// pipe (2400 triangles in 13 x 13 x 34 cells), of 0.05 / 0.5 / 1 / 2 / 8 of a cell's size, us:
// cells alone 41 / 84 / 116 / 221 / 1747, segment grid alone 32 / 76 / 182 / 605 / 12787,
// with 4 / 8 / 16 / 64 visits at most 31 88 118 226 1761 / 32 90 124 223 1746 / 31 81 158
// 227 1760 / 32 78 179 344 1772; with a loop for each grid and 8, which spills less in
// the tracks' kernels, 31 91 106 191 1522.
constexpr int kSegMostVisits = 8;

__device__ __forceinline__ bool segment_hits_surface(const SurfaceDev& S, V3 p0, V3 p1) {
    const double a0[3] = {p0.x, p0.y, p0.z}, a1[3] = {p1.x, p1.y, p1.z};
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u0 = (fmin(a0[a], a1[a]) - S.lo[a]) * S.seg_inv_h[a];
        const double u1 = (fmax(a0[a], a1[a]) - S.lo[a]) * S.seg_inv_h[a];
        if (!(u1 >= 0.0 && u0 < (double)S.seg_dims[a])) return false;   // beyond the mesh (or NaN)
        lo[a] = u0 <= 0.0 ? 0 : (int)u0;
        hi[a] = u1 >= (double)(S.seg_dims[a] - 1) ? S.seg_dims[a] - 1 : (int)u1;
    }
    const V3 d = v3(__dsub_rn(p1.x, p0.x), __dsub_rn(p1.y, p0.y), __dsub_rn(p1.z, p0.z));
    const V3 centre = v3(S.centre[0], S.centre[1], S.centre[2]);
    const V3 from = p0 - centre, to = p1 - centre;
    const double margin = 0x1p-43 * (S.reach + fabs(from.x) + fabs(from.y) + fabs(from.z) + fabs(to.x) + fabs(to.y) +
                                     fabs(to.z));
    const bool many = (hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1) > kSegMostVisits;
    if (!many) return cells_hit(S, S.seg_start, S.seg_tri, S.seg_dims[1], S.seg_dims[2], lo, hi, p0, d, from, to, margin);
    const int parts = S.seg_dims[0] / S.dims[0];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] /= parts;
        hi[a] /= parts;
    }
    return cells_hit(S, S.cell_start, S.cell_tri, S.dims[1], S.dims[2], lo, hi, p0, d, from, to, margin);
}

// A box around a point in which no segment can meet the surface: the cells
// closer than the nearest one that lists a triangle (clearance), or the part of
// such a cell whose segment-grid cell lists none, or, beyond the
// grid, everything beyond it on that side.  A tracked particle whose step ends
// in the box it started in needs no test; it takes six comparisons where the
// test takes some sixty instructions without a triangle in sight.  The box is
// kept a millionth of a cell inside its cells, far more than the rounding of the
// test's cell index, so a step it lets pass is one the test would have passed.
struct ClearBox {
    V3 lo, hi;
};

__device__ __forceinline__ ClearBox no_clear_box() {
    return ClearBox{v3(INFINITY, INFINITY, INFINITY), v3(-INFINITY, -INFINITY, -INFINITY)};
}

__device__ __forceinline__ bool in_clear_box(const ClearBox& b, V3 p) {
    return (p.x >= b.lo.x) & (p.x <= b.hi.x) & (p.y >= b.lo.y) & (p.y <= b.hi.y) & (p.z >= b.lo.z) & (p.z <= b.hi.z);
}

__device__ __forceinline__ ClearBox clear_box(const SurfaceDev& S, V3 p) {
    if (S.clearance == nullptr) return no_clear_box();
    const double pc[3] = {p.x, p.y, p.z};
    double lo[3], hi[3];
    int cell[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u = (pc[a] - S.lo[a]) * S.inv_h[a];
        if (!(u == u)) return no_clear_box();
        cell[a] = u < 0.0 ? -1 : (u >= (double)S.dims[a] ? S.dims[a] : (int)u);
        lo[a] = -INFINITY;
        hi[a] = INFINITY;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double m = 1e-6 * S.h[a];
        if (cell[a] < 0) {
            hi[a] = S.lo[a] - m;
            return ClearBox{v3(lo[0], lo[1], lo[2]), v3(hi[0], hi[1], hi[2])};
        }
        if (cell[a] >= S.dims[a]) {
            lo[a] = S.lo[a] + S.dims[a] * S.h[a] + m;
            return ClearBox{v3(lo[0], lo[1], lo[2]), v3(hi[0], hi[1], hi[2])};
        }
    }
    const int c = S.clearance[(cell[0] * S.dims[1] + cell[1]) * S.dims[2] + cell[2]];
    if (c == 0) {
        // next to the surface: the segment grid's cell, if that lists nothing
        int s[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int at = (int)((pc[a] - S.lo[a]) * S.seg_inv_h[a]);
            s[a] = at < S.seg_dims[a] ? at : S.seg_dims[a] - 1;
            const double m = 1e-6 * S.seg_h[a];
            lo[a] = S.lo[a] + s[a] * S.seg_h[a] + m;
            hi[a] = S.lo[a] + (s[a] + 1) * S.seg_h[a] - m;
        }
        const int at = (s[0] * S.seg_dims[1] + s[1]) * S.seg_dims[2] + s[2];
        if (S.seg_start[at + 1] > S.seg_start[at]) return no_clear_box();
        return ClearBox{v3(lo[0], lo[1], lo[2]), v3(hi[0], hi[1], hi[2])};
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // cells cell - (c - 1) .. cell + (c - 1) list nothing; nothing lies beyond the grid either
        const double m = 1e-6 * S.h[a];
        if (cell[a] - (c - 1) > 0) lo[a] = S.lo[a] + (cell[a] - (c - 1)) * S.h[a] + m;
        if (cell[a] + c < S.dims[a]) hi[a] = S.lo[a] + (cell[a] + c) * S.h[a] - m;
    }
    return ClearBox{v3(lo[0], lo[1], lo[2]), v3(hi[0], hi[1], hi[2])};
}

// Steps of d (per step) a point in the box certainly stays in it.
__device__ __forceinline__ int clear_steps(const ClearBox& b, V3 p, V3 d) {
    const double x[3] = {p.x, p.y, p.z}, u[3] = {d.x, d.y, d.z};
    const double lo[3] = {b.lo.x, b.lo.y, b.lo.z}, hi[3] = {b.hi.x, b.hi.y, b.hi.z};
    double k = 1e9;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (u[a] != 0.0) k = fmin(k, u[a] > 0.0 ? (hi[a] - x[a]) / u[a] : (lo[a] - x[a]) / u[a]);
    k = k * (1.0 - 1e-9) - 1.0;
    return k >= 1.0 ? (int)k : 0;      // (a point that is NaN has no clear box, whose infinities give 0)
}

// Ray p + t d (t >= 0) against one triangle: the hit's t, or -1.  The same
// rounded operations as segment_hits_triangle.
__device__ __forceinline__ double ray_triangle_t(const double* __restrict__ T, V3 p0, V3 d) {
    const V3 v0 = v3(T[0], T[1], T[2]);
    const V3 e1 = v3(T[3], T[4], T[5]);
    const V3 e2 = v3(T[6], T[7], T[8]);
    const V3 pv = rn_cross(d, e2);
    const double det = rn_dot(e1.x, e1.y, e1.z, pv.x, pv.y, pv.z);
    if (det == 0.0) return -1.0;
    const double inv = 1.0 / det;
    const V3 tv = v3(__dsub_rn(p0.x, v0.x), __dsub_rn(p0.y, v0.y), __dsub_rn(p0.z, v0.z));
    const double u = __dmul_rn(rn_dot(tv.x, tv.y, tv.z, pv.x, pv.y, pv.z), inv);
    if (!(u >= 0.0 && u <= 1.0)) return -1.0;
    const V3 qv = rn_cross(tv, e1);
    const double v = __dmul_rn(rn_dot(d.x, d.y, d.z, qv.x, qv.y, qv.z), inv);
    if (!(v >= 0.0 && __dadd_rn(u, v) <= 1.0)) return -1.0;
    const double t = __dmul_rn(rn_dot(e2.x, e2.y, e2.z, qv.x, qv.y, qv.z), inv);
    return t >= 0.0 ? t : -1.0;
}

// Crossings of the axis-parallel ray from p in direction dir (0..5 = +x -x
// +y -y +z -z) with the surface: their number and the nearest one's distance
// (INFINITY without any).  The ray walks the column of grid cells it lies in;
// a triangle listed in several cells of the column is tested in the first of
// them the walk reaches.
__device__ __forceinline__ void axis_ray_hits(const SurfaceDev& S, V3 p, int dir, int& count, double& dist) {
    const int ax = dir >> 1;
    const double sgn = (dir & 1) ? -1.0 : 1.0;
    const double pc[3] = {p.x, p.y, p.z};
    count = 0;
    dist = INFINITY;
    int cell[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u = (pc[a] - S.lo[a]) * S.inv_h[a];
        if (!(u == u)) return;                                            // NaN
        if (a != ax && !(u >= 0.0 && u < (double)S.dims[a])) return;   // the column misses the mesh
        cell[a] = u < 0.0 ? -1 : (u >= (double)S.dims[a] ? S.dims[a] : (int)u);
    }
    const V3 d = v3(ax == 0 ? sgn : 0.0, ax == 1 ? sgn : 0.0, ax == 2 ? sgn : 0.0);
    int c0 = cell[ax], step = (dir & 1) ? -1 : 1;
    if (step > 0) c0 = c0 < 0 ? 0 : c0;
    else c0 = c0 >= S.dims[ax] ? S.dims[ax] - 1 : c0;
    for (int c = c0; c >= 0 && c < S.dims[ax]; c += step) {
        cell[ax] = c;
        const int lin = (cell[0] * S.dims[1] + cell[1]) * S.dims[2] + cell[2];
        const int end = S.cell_start[lin + 1];
        for (int q = S.cell_start[lin]; q < end; ++q) {
            const int tri = S.cell_tri[q];
            const int lo = S.trange[6 * tri + 2 * ax], hi = S.trange[6 * tri + 2 * ax + 1];
            const int first = step > 0 ? (c0 > lo ? c0 : lo) : (c0 < hi ? c0 : hi);
            if (c != first) continue;     // tested in an earlier cell of the walk
            const double t = ray_triangle_t(S.tri + 9 * (int64_t)tri, p, d);
            if (t >= 0.0) {
                ++count;
                dist = t < dist ? t : dist;
            }
        }
    }
}

}  // namespace ppt

struct ppt_surface {
    int device;
    ppt::SurfaceDev dev;
    void* buf;          // one device allocation: triangles, cell offsets, cell lists
    void* seg_buf;      // the segment grid's and the clearances', once refined
    size_t bytes;
    std::vector<int32_t> start;  // the cells' list offsets
    std::vector<double> boxes;   // the triangles' bounding boxes (lo x y z, hi x y z)
    std::mutex refining;         // one ppt_surface_refine at a time
    mutable std::mutex m;        // dev and bytes, which it changes while other threads use the surface
    ppt::SurfaceDev view() const {
        std::lock_guard<std::mutex> lock(m);
        return dev;
    }
};
