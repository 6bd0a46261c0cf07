// Electrode surfaces: upload of a triangle mesh with its cell grid, and the
// standalone segment test (the call the reference makes each step,
// PyElectrodeAssembly.segment_intersects_surface, src/PyPATools/pusher.py:984).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "surface.cuh"

namespace ppt {

__global__ void segments_hit_kernel(const __grid_constant__ SurfaceDev S, int64_t n, const double* __restrict__ p0,
                                    const double* __restrict__ p1, uint8_t* __restrict__ hit) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V3 a = v3(p0[3 * i], p0[3 * i + 1], p0[3 * i + 2]);
    const V3 b = v3(p1[3 * i], p1[3 * i + 1], p1[3 * i + 2]);
    hit[i] = segment_hits_surface(S, a, b) ? 1 : 0;
}

// Cell grid over the mesh's bounding box: about two cells per triangle, cells
// as close to cubes as the box allows, at most 256 per axis.
static void grid_for_mesh(const double lo_in[3], const double hi_in[3], int64_t n_tri, double lo[3],
                          double h[3], int dims[3]) {
    double ext[3], big = 0.0;
    for (int a = 0; a < 3; ++a) big = std::max(big, hi_in[a] - lo_in[a]);
    const double pad = std::max(big * 1e-9, 1e-30);
    double vol = 1.0;
    for (int a = 0; a < 3; ++a) {
        lo[a] = lo_in[a] - pad;
        ext[a] = (hi_in[a] + pad) - lo[a];
        vol *= ext[a];
    }
    const double target = std::max<double>(1.0, 2.0 * (double)n_tri);
    const double side = std::cbrt(vol / target);
    for (int a = 0; a < 3; ++a) {
        double d = std::ceil(ext[a] / side);
        d = d < 1.0 ? 1.0 : (d > 256.0 ? 256.0 : d);
        dims[a] = (int)d;
        h[a] = ext[a] / (double)dims[a];
    }
}

// Distance of every cell to the nearest one that lists a triangle, in cells
// along the farthest axis (two passes over the 26 neighbours), at most 255.
static std::vector<uint8_t> cell_clearance(const int dims[3], const std::vector<int32_t>& start) {
    const int64_t cells = (int64_t)dims[0] * dims[1] * dims[2];
    std::vector<uint8_t> c((size_t)cells);
    for (int64_t i = 0; i < cells; ++i) c[(size_t)i] = start[(size_t)i + 1] > start[(size_t)i] ? 0 : 255;
    for (int pass = 0; pass < 2; ++pass) {
        const int way = pass == 0 ? -1 : 1;
        for (int64_t n = 0; n < cells; ++n) {
            const int64_t at = pass == 0 ? n : cells - 1 - n;
            const int k = (int)(at % dims[2]), j = (int)(at / dims[2] % dims[1]), i = (int)(at / dims[2] / dims[1]);
            int best = c[(size_t)at];
            for (int di = 0; di <= 1 && best > 0; ++di)
                for (int dj = di ? -1 : 0; dj <= 1; ++dj)
                    for (int dk = di || dj ? -1 : 1; dk <= 1; ++dk) {
                        // the 13 neighbours that the pass has been at
                        const int ni = i + way * di, nj = j + way * dj, nk = k + way * dk;
                        if (ni < 0 || ni >= dims[0] || nj < 0 || nj >= dims[1] || nk < 0 || nk >= dims[2]) continue;
                        const int far = c[(size_t)(((int64_t)ni * dims[1] + nj) * dims[2] + nk)] + 1;
                        best = far < best ? far : best;
                    }
            c[(size_t)at] = (uint8_t)best;
        }
    }
    return c;
}

// Bin each triangle into the cells its bounding box overlaps (count, then
// fill); false when the lists exceed 2^31 entries.  The box is padded by 1e-7 of
// a cell: the segment and ray tests work on v0, e1 = v1 - v0, e2 = v2 - v0
// rounded, whose hits can lie an ulp or so outside the vertices' box; a triangle
// within the pad of a cell face is listed on both sides of it, so no such hit
// falls in a cell that does not list the triangle (the tests stay the same as
// testing every triangle).
static bool bin_triangles(const ppt_surface& S, const double inv_h[3], const int32_t dims[3],
                          std::vector<int32_t>* start, std::vector<int32_t>* list, std::vector<int32_t>* range) {
    const int64_t n_tri = (int64_t)S.boxes.size() / 6;
    const int64_t cells = (int64_t)dims[0] * dims[1] * dims[2];
    auto cell_range = [&](int64_t t, int r0[3], int r1[3]) {
        for (int a = 0; a < 3; ++a) {
            const double pad = 1e-7 / inv_h[a];
            const double u0 = (S.boxes[6 * t + a] - pad - S.dev.lo[a]) * inv_h[a];
            const double u1 = (S.boxes[6 * t + 3 + a] + pad - S.dev.lo[a]) * inv_h[a];
            r0[a] = std::min(std::max((int)std::floor(u0), 0), dims[a] - 1);
            r1[a] = std::min(std::max((int)std::floor(u1), 0), dims[a] - 1);
        }
    };
    std::vector<int64_t> count((size_t)cells + 1, 0);
    if (range) range->resize((size_t)n_tri * 6);
    for (int64_t t = 0; t < n_tri; ++t) {
        int r0[3], r1[3];
        cell_range(t, r0, r1);
        if (range)
            for (int a = 0; a < 3; ++a) {
                (*range)[6 * t + 2 * a] = r0[a];
                (*range)[6 * t + 2 * a + 1] = r1[a];
            }
        for (int i = r0[0]; i <= r1[0]; ++i)
            for (int j = r0[1]; j <= r1[1]; ++j)
                for (int k = r0[2]; k <= r1[2]; ++k) ++count[(i * (int64_t)dims[1] + j) * dims[2] + k + 1];
    }
    for (int64_t c = 0; c < cells; ++c) count[c + 1] += count[c];
    if (count[cells] > 0x7fffffffLL) return false;
    start->assign(count.begin(), count.end());
    list->resize((size_t)count[cells]);
    std::vector<int32_t> fill(start->begin(), start->end() - 1);
    for (int64_t t = 0; t < n_tri; ++t) {
        int r0[3], r1[3];
        cell_range(t, r0, r1);
        for (int i = r0[0]; i <= r1[0]; ++i)
            for (int j = r0[1]; j <= r1[1]; ++j)
                for (int k = r0[2]; k <= r1[2]; ++k)
                    (*list)[fill[(i * (int64_t)dims[1] + j) * dims[2] + k]++] = (int32_t)t;
    }
    return true;
}

}  // namespace ppt

using namespace ppt;

extern "C" int ppt_surface_create(int64_t n_vertices, const double* vertices, int64_t n_triangles,
                                  const int64_t* triangles, ppt_surface** out) {
    if (!out) return fail(PPT_ERR_ARG, "out must not be NULL");
    *out = nullptr;
    if (n_vertices < 3 || n_triangles < 1) return fail(PPT_ERR_ARG, "a surface needs >= 3 vertices and >= 1 triangle");
    if (!vertices || !triangles) return fail(PPT_ERR_ARG, "vertices and triangles must not be NULL");
    if (n_triangles > (1LL << 30)) return fail(PPT_ERR_ARG, "too many triangles");
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    std::vector<double> tri((size_t)n_triangles * 9);
    for (int64_t t = 0; t < n_triangles; ++t) {
        const double* v[3];
        for (int c = 0; c < 3; ++c) {
            const int64_t idx = triangles[3 * t + c];
            if (idx < 0 || idx >= n_vertices) return fail(PPT_ERR_ARG, "triangle vertex index out of range");
            v[c] = vertices + 3 * idx;
        }
        for (int a = 0; a < 3; ++a) {
            for (int c = 0; c < 3; ++c) {
                if (!std::isfinite(v[c][a])) return fail(PPT_ERR_ARG, "vertex coordinates must be finite");
                lo[a] = std::min(lo[a], v[c][a]);
                hi[a] = std::max(hi[a], v[c][a]);
            }
            tri[9 * t + a] = v[0][a];
            tri[9 * t + 3 + a] = v[1][a] - v[0][a];
            tri[9 * t + 6 + a] = v[2][a] - v[0][a];
        }
    }
    std::unique_ptr<ppt_surface> own(new (std::nothrow) ppt_surface());
    if (!own) return fail(PPT_ERR_OOM, "surface handle");
    ppt_surface& S = *own;
    std::memset(&S.dev, 0, sizeof(S.dev));
    double h[3];
    grid_for_mesh(lo, hi, n_triangles, S.dev.lo, h, S.dev.dims);
    for (int a = 0; a < 3; ++a) {
        S.dev.inv_h[a] = 1.0 / h[a];
        S.dev.h[a] = h[a];
    }
    S.boxes.resize((size_t)n_triangles * 6);
    for (int64_t t = 0; t < n_triangles; ++t)
        for (int a = 0; a < 3; ++a) {
            const double x[3] = {vertices[3 * triangles[3 * t] + a], vertices[3 * triangles[3 * t + 1] + a],
                                 vertices[3 * triangles[3 * t + 2] + a]};
            S.boxes[6 * t + a] = std::min(x[0], std::min(x[1], x[2]));
            S.boxes[6 * t + 3 + a] = std::max(x[0], std::max(x[1], x[2]));
        }
    std::vector<int32_t> start, list, trange;
    if (!bin_triangles(S, S.dev.inv_h, S.dev.dims, &start, &list, &trange))
        return fail(PPT_ERR_UNSUPPORTED, "surface cell lists exceed 2^31 entries");
    double reach = 0.0;
    for (int a = 0; a < 3; ++a) {
        const double half = 0.5 * h[a] * S.dev.dims[a];
        S.dev.centre[a] = S.dev.lo[a] + half;
        reach += half;
    }
    S.dev.reach = reach;
    // planes after the triangles, at 32 bytes each (one load)
    const size_t tri_end = (tri.size() + 3) / 4 * 4;
    tri.resize(tri_end + (size_t)n_triangles * 4);
    for (int64_t t = 0; t < n_triangles; ++t) {
        const double* v = &tri[9 * (size_t)t];
        const double* e = v + 3;
        const double* f = v + 6;
        const double size = std::sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]) *
                            std::sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
        double* p = &tri[tri_end + 4 * (size_t)t];
        const double n[3] = {e[1] * f[2] - e[2] * f[1], e[2] * f[0] - e[0] * f[2], e[0] * f[1] - e[1] * f[0]};
        p[3] = 0.0;
        for (int a = 0; a < 3; ++a) {
            // (a triangle without area keeps a plane that decides nothing)
            p[a] = size > 0.0 ? n[a] / size : 0.0;
            p[3] -= p[a] * (v[a] - S.dev.centre[a]);
        }
    }
    const size_t b_tri = tri.size() * sizeof(double);
    const size_t b_start = start.size() * sizeof(int32_t);
    const size_t b_list = std::max<size_t>(list.size(), 1) * sizeof(int32_t);
    const size_t b_range = trange.size() * sizeof(int32_t);
    S.bytes = b_tri + b_start + b_list + b_range;
    PPT_CUDA_TRY(cudaGetDevice(&S.device));
    cudaError_t e = cudaMalloc(&S.buf, S.bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(PPT_ERR_OOM, "cudaMalloc of the surface failed");
    }
    char* base = static_cast<char*>(S.buf);
    e = cudaMemcpy(base, tri.data(), b_tri, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(base + b_tri, start.data(), b_start, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !list.empty())
        e = cudaMemcpy(base + b_tri + b_start, list.data(), list.size() * sizeof(int32_t), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(base + b_tri + b_start + b_list, trange.data(), b_range, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(S.buf);
        return cuda_fail(e, "surface upload");
    }
    S.dev.tri = reinterpret_cast<const double*>(base);
    S.dev.plane = reinterpret_cast<const double*>(base) + tri_end;
    S.dev.cell_start = reinterpret_cast<const int32_t*>(base + b_tri);
    S.dev.cell_tri = reinterpret_cast<const int32_t*>(base + b_tri + b_start);
    S.dev.trange = reinterpret_cast<const int32_t*>(base + b_tri + b_start + b_list);
    S.start = std::move(start);
    S.dev.n_tri = (int32_t)n_triangles;
    S.dev.seg_start = S.dev.cell_start;
    S.dev.seg_tri = S.dev.cell_tri;
    for (int a = 0; a < 3; ++a) {
        S.dev.seg_h[a] = h[a];
        S.dev.seg_inv_h[a] = S.dev.inv_h[a];
        S.dev.seg_dims[a] = S.dev.dims[a];
    }
    *out = own.release();
    return PPT_OK;
}

// Segment-grid cells per axis of a cell, and the most cells such a grid may
// have.  A particle within a cell of a wall tests the triangles its cell lists at
// every step; finer cells list fewer and leave more of the space near the wall
// clear.  1e6 protons x 1000 steps through a pipe and an aperture plate (2400
// triangles, 5746 cells), kernel time: the cells themselves 10.6 ms, with 2 / 3 / 4 /
// 6 parts per axis 8.1 / 7.6 / 7.5 / 7.2 (15.1 before the plane and box tests).
constexpr int kSegFactor = 4;
constexpr int64_t kSegMostCells = 1 << 21;

extern "C" int ppt_surface_refine(ppt_surface* s) {
    if (!s) return fail(PPT_ERR_ARG, "surface is NULL");
    try {
        std::lock_guard<std::mutex> one(s->refining);
        if (s->seg_buf) return PPT_OK;
        SurfaceDev D = s->dev;
        const std::vector<uint8_t> clearance = cell_clearance(D.dims, s->start);
        const int64_t cells = (int64_t)clearance.size();
        int f = kSegFactor;
        while (f > 1 && cells * f * f * f > kSegMostCells) --f;
        for (int a = 0; a < 3; ++a) {
            D.seg_dims[a] = D.dims[a] * f;
            D.seg_h[a] = D.h[a] / f;
            D.seg_inv_h[a] = D.inv_h[a] * f;
        }
        std::vector<int32_t> start, list;
        // (the cells themselves when the lists would be too long)
        if (f > 1 && !bin_triangles(*s, D.seg_inv_h, D.seg_dims, &start, &list, nullptr)) f = 1;
        const size_t b_start = f > 1 ? start.size() * sizeof(int32_t) : 0;
        const size_t b_list = f > 1 ? list.size() * sizeof(int32_t) : 0;
        int prev = 0;
        PPT_CUDA_TRY(cudaGetDevice(&prev));
        PPT_CUDA_TRY(cudaSetDevice(s->device));
        void* buf = nullptr;
        cudaError_t e = cudaMalloc(&buf, b_start + b_list + clearance.size());
        char* base = static_cast<char*>(buf);
        if (e == cudaSuccess && b_start) e = cudaMemcpy(base, start.data(), b_start, cudaMemcpyHostToDevice);
        if (e == cudaSuccess && b_list) e = cudaMemcpy(base + b_start, list.data(), b_list, cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
            e = cudaMemcpy(base + b_start + b_list, clearance.data(), clearance.size(), cudaMemcpyHostToDevice);
        cudaSetDevice(prev);
        if (e != cudaSuccess) {
            cudaGetLastError();
            if (buf) cudaFree(buf);
            return e == cudaErrorMemoryAllocation ? fail(PPT_ERR_OOM, "cudaMalloc of the segment grid failed")
                                                  : cuda_fail(e, "segment grid upload");
        }
        std::lock_guard<std::mutex> lock(s->m);
        s->dev.clearance = reinterpret_cast<const uint8_t*>(base + b_start + b_list);
        if (f > 1) {
            D.clearance = s->dev.clearance;
            D.seg_start = reinterpret_cast<const int32_t*>(base);
            D.seg_tri = D.seg_start + start.size();
            s->dev = D;
        }
        s->seg_buf = buf;
        s->bytes += b_start + b_list + clearance.size();
        return PPT_OK;
    } catch (const std::exception& ex) {
        return fail(PPT_ERR_OOM, std::string("segment grid: ") + ex.what());
    }
}

__global__ void axis_rays_kernel(const __grid_constant__ SurfaceDev S, int64_t n, const double* __restrict__ pts,
                                 double* __restrict__ dist, int32_t* __restrict__ hits) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n * 6) return;
    const int64_t row = i / 6;
    const int dir = (int)(i - row * 6);
    int c;
    double d;
    axis_ray_hits(S, v3(pts[3 * row], pts[3 * row + 1], pts[3 * row + 2]), dir, c, d);
    dist[i] = d;
    hits[i] = c;
}

extern "C" int ppt_surface_axis_rays(const ppt_surface* s, int64_t n, const double* points, double* min_dist,
                                     int32_t* hits, void* stream) {
    if (!s) return fail(PPT_ERR_ARG, "surface is NULL");
    if (n < 0) return fail(PPT_ERR_ARG, "n must be >= 0");
    if (n == 0) return PPT_OK;
    if (!points || !min_dist || !hits) return fail(PPT_ERR_ARG, "points, min_dist and hits must not be NULL");
    const int block = 128;
    axis_rays_kernel<<<grid_for(n * 6, block), block, 0, static_cast<cudaStream_t>(stream)>>>(s->view(), n, points,
                                                                                              min_dist, hits);
    PPT_CUDA_TRY(cudaGetLastError());
    return PPT_OK;
}

extern "C" int ppt_surface_destroy(ppt_surface* s) {
    if (!s) return PPT_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(s->device);
    cudaError_t e = cudaFree(s->buf);
    if (s->seg_buf) {
        const cudaError_t e2 = cudaFree(s->seg_buf);
        if (e == cudaSuccess) e = e2;
    }
    cudaSetDevice(prev);
    delete s;
    if (e != cudaSuccess) return cuda_fail(e, "cudaFree(surface)");
    return PPT_OK;
}

extern "C" int ppt_surface_info(const ppt_surface* s, int64_t* bytes, int32_t dims[3]) {
    if (!s) return fail(PPT_ERR_ARG, "surface is NULL");
    std::lock_guard<std::mutex> lock(s->m);
    if (bytes) *bytes = (int64_t)s->bytes;
    if (dims)
        for (int a = 0; a < 3; ++a) dims[a] = s->dev.dims[a];
    return PPT_OK;
}

extern "C" int ppt_surface_segments_hit(const ppt_surface* s, int64_t n, const double* p0, const double* p1,
                                        uint8_t* hit, void* stream) {
    if (!s) return fail(PPT_ERR_ARG, "surface is NULL");
    if (n < 0) return fail(PPT_ERR_ARG, "n must be >= 0");
    if (n == 0) return PPT_OK;
    if (!p0 || !p1 || !hit) return fail(PPT_ERR_ARG, "p0, p1 and hit must not be NULL");
    const int block = 128;
    segments_hit_kernel<<<grid_for(n, block), block, 0, static_cast<cudaStream_t>(stream)>>>(s->view(), n, p0, p1,
                                                                                             hit);
    PPT_CUDA_TRY(cudaGetLastError());
    return PPT_OK;
}
