// Space-charge potential and field on the Poisson solver's mesh.
//
// Reference: PyAMGPoissonSolver (src/PyPATools/poisson_amg.py).  Its mesh has
// n[a] cells of size h = extent / n centred at -extent/2 + (i + 1/2) h
// (:227-239); the operator is the 7-point Laplacian assembled at :293-443,
// which without conductor cells is, per axis, 2 / (h h) on the diagonal and
// -2 / (h (h + h)) for each neighbour inside the box (a neighbour beyond the
// box is a zero potential one cell away); the right-hand side is rho / eps0
// (:913-921).  The reference solves with GMRES preconditioned by an AMG
// V-cycle to a relative residual (1e-6 by default, :70); here the operator is
// applied matrix-free and the system, symmetric positive definite, is solved
// by conjugate gradients to the requested relative residual.  E = -grad phi by
// central differences at the cells whose three indices are all interior,
// zero on the outer layer (compute_field_from_potential_numba, :98-130).
//
// Every reduction sums per-block partials in a fixed order (no atomics), and
// the iteration stops on the device at the first iterate meeting the
// tolerance: a solve gives the same bits however its launches are batched.
#include <cmath>

#include "ppt_internal.cuh"

namespace ppt {

struct PoissonOp {
    int64_t n[3];
    double off[3];   // the neighbour coefficients, -2 / (h (h + h)) per axis
    double diag;     // 2/(hx hx) + 2/(hy hy) + 2/(hz hz), summed in that order from 0
};

// Scalars the kernels share, in device memory.
enum { kRR = 0, kALPHA, kBETA, kDONE, kITERS, kTOL2, kBB, kNumScalars };

constexpr int kBlock = 256;

__device__ __forceinline__ double apply_op(const PoissonOp& A, const double* __restrict__ x, int64_t c, int64_t i,
                                           int64_t j, int64_t k) {
    const int64_t sy = A.n[2], sx = A.n[1] * A.n[2];
    double s = A.diag * x[c];
    // x, y, z neighbours as the reference's rows list them
    if (i + 1 < A.n[0]) s += A.off[0] * x[c + sx];
    if (i > 0) s += A.off[0] * x[c - sx];
    if (j + 1 < A.n[1]) s += A.off[1] * x[c + sy];
    if (j > 0) s += A.off[1] * x[c - sy];
    if (k + 1 < A.n[2]) s += A.off[2] * x[c + 1];
    if (k > 0) s += A.off[2] * x[c - 1];
    return s;
}

// Block sum of v into partial[blockIdx.x] (fixed shuffle / shared order).
__device__ __forceinline__ void block_partial(double v, double* partial) {
    __shared__ double warp_sums[kBlock / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kBlock / 32; ++w) s += warp_sums[w];
        partial[blockIdx.x] = s;
    }
}

__device__ __forceinline__ void cell_ijk(const PoissonOp& A, int64_t c, int64_t& i, int64_t& j, int64_t& k) {
    k = c % A.n[2];
    const int64_t t = c / A.n[2];
    j = t % A.n[1];
    i = t / A.n[1];
}

// r = b - A x, p = r; partial sums of r.r and b.b
__global__ void __launch_bounds__(kBlock) cg_start(const __grid_constant__ PoissonOp A, int64_t m,
                                                   const double* __restrict__ b, const double* __restrict__ x,
                                                   double* __restrict__ r, double* __restrict__ p,
                                                   double* __restrict__ part_rr, double* __restrict__ part_bb) {
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double rr = 0.0, bb = 0.0;
    if (c < m) {
        int64_t i, j, k;
        cell_ijk(A, c, i, j, k);
        const double rc = b[c] - apply_op(A, x, c, i, j, k);
        r[c] = rc;
        p[c] = rc;
        rr = rc * rc;
        bb = b[c] * b[c];
    }
    block_partial(rr, part_rr);
    __syncthreads();
    block_partial(bb, part_bb);
}

// q = A p; partial sums of p.q
__global__ void __launch_bounds__(kBlock) cg_apply(const __grid_constant__ PoissonOp A, int64_t m,
                                                   const double* __restrict__ p, double* __restrict__ q,
                                                   double* __restrict__ part, const double* __restrict__ S) {
    if (S[kDONE] != 0.0) return;
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double s = 0.0;
    if (c < m) {
        int64_t i, j, k;
        cell_ijk(A, c, i, j, k);
        const double qc = apply_op(A, p, c, i, j, k);
        q[c] = qc;
        s = p[c] * qc;
    }
    block_partial(s, part);
}

// x += alpha p, r -= alpha q; partial sums of r.r
__global__ void __launch_bounds__(kBlock) cg_step(int64_t m, double* __restrict__ x, double* __restrict__ r,
                                                  const double* __restrict__ p, const double* __restrict__ q,
                                                  double* __restrict__ part, const double* __restrict__ S) {
    if (S[kDONE] != 0.0) return;
    const double alpha = S[kALPHA];
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double s = 0.0;
    if (c < m) {
        x[c] += alpha * p[c];
        const double rc = r[c] - alpha * q[c];
        r[c] = rc;
        s = rc * rc;
    }
    block_partial(s, part);
}

// p = r + beta p
__global__ void __launch_bounds__(kBlock) cg_direction(int64_t m, const double* __restrict__ r, double* __restrict__ p,
                                                       const double* __restrict__ S) {
    if (S[kDONE] != 0.0) return;
    const double beta = S[kBETA];
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (c < m) p[c] = r[c] + beta * p[c];
}

__device__ double sum_partials(const double* part, int nb) {
    __shared__ double s[kBlock];
    double v = 0.0;
    for (int b = threadIdx.x; b < nb; b += kBlock) v += part[b];
    s[threadIdx.x] = v;
    __syncthreads();
    for (int w = kBlock / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    return s[0];
}

// One block.  mode 0: start (rr, bb -> tolerance); 1: alpha = rr / p.q;
// 2: rr' and beta = rr' / rr, stop once rr' <= tol^2 bb or rr' = 0.
__global__ void __launch_bounds__(kBlock) cg_scalars(int mode, const double* __restrict__ part,
                                                     const double* __restrict__ part2, int nb, double* S,
                                                     double rel_tol, int64_t max_iter) {
    if (mode != 0 && S[kDONE] != 0.0) return;
    const double v = sum_partials(part, nb);
    __syncthreads();
    if (mode == 0) {
        const double bb = sum_partials(part2, nb);
        if (threadIdx.x == 0) {
            S[kRR] = v;
            S[kBB] = bb;
            S[kTOL2] = rel_tol * rel_tol * bb;
            S[kITERS] = 0.0;
            S[kDONE] = (v <= S[kTOL2] || v == 0.0 || max_iter <= 0) ? 1.0 : 0.0;
        }
        return;
    }
    if (threadIdx.x != 0) return;
    if (mode == 1) {
        S[kALPHA] = S[kRR] / v;
    } else {
        S[kBETA] = v / S[kRR];
        S[kRR] = v;
        S[kITERS] += 1.0;
        if (v <= S[kTOL2] || v == 0.0 || S[kITERS] >= (double)max_iter) S[kDONE] = 1.0;
    }
}

__global__ void __launch_bounds__(kBlock) field_from_potential(int64_t nx, int64_t ny, int64_t nz,
                                                               const double* __restrict__ phi, double hx, double hy,
                                                               double hz, double* __restrict__ ex,
                                                               double* __restrict__ ey, double* __restrict__ ez) {
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (c >= nx * ny * nz) return;
    const int64_t k = c % nz, t = c / nz, j = t % ny, i = t / ny;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (i > 0 && i < nx - 1 && j > 0 && j < ny - 1 && k > 0 && k < nz - 1) {
        const int64_t sy = nz, sx = ny * nz;
        fx = -(phi[c + sx] - phi[c - sx]) / (2 * hx);
        fy = -(phi[c + sy] - phi[c - sy]) / (2 * hy);
        fz = -(phi[c + 1] - phi[c - 1]) / (2 * hz);
    }
    if (ex) ex[c] = fx;
    if (ey) ey[c] = fy;
    if (ez) ez[c] = fz;
}

// ---------------------------------------------------------------------------
// Operator with per-cell coefficients (conductor cells, Shortley-Weller rows):
// coef[7 c .. 7 c + 6] = diagonal, +x, -x, +y, -y, +z, -z couplings (0 for a
// neighbour outside the box or in a conductor; a conductor cell's row is the
// identity).  Not symmetric in general: BiCGSTAB (H. A. van der Vorst, SIAM J.
// Sci. Stat. Comput. 13(2), 1992).
// ---------------------------------------------------------------------------
struct CoefOp {
    int64_t n[3];
    const double* coef;
};

enum { bRR = 0, bBB, bTOL2, bRHO, bRHAT2, bALPHA, bOMEGA, bBETA, bFRESH, bDONE, bITERS, bNumScalars };

// Both forms of the iteration below (launched here, in one kernel further down)
// have the diagonal as right preconditioner: A is applied to p^ = p / d and
// s^ = s / d, and the residual and the stopping test stay those of the rows as they
// are.  A row next to a conductor surface a thousandth of a cell away has entries up
// to 1000 times the others'; without the division the iteration spends most of its
// steps on them, and its rhat.r can vanish to rounding before it converges
// (64 x 64 x 128 cells, pipe and aperture: 370-450 iterations to 1e-6, with it about
// 140; 36 x 59 x 117 to 1e-8: stopped at residuals between 4e-9 and 0.16, with it 141
// iterations).  Once rho = rhat.r is within the rounding of its sum, the iteration
// starts again from r as its rhat.
constexpr double kRhoRounding = 1e-28;     // (1e-14)^2, of |rhat|^2 |r|^2

// The diagonal, or 1 where it cannot be divided by.
__device__ __forceinline__ double row_scale(double diag) {
    return diag != 0.0 && isfinite(1.0 / diag) ? diag : 1.0;
}

__device__ __forceinline__ double apply_coef(const CoefOp& A, const double* __restrict__ x, int64_t c) {
    const int64_t nz = A.n[2], sy = nz, sx = A.n[1] * nz;
    const int64_t k = c % nz, t = c / nz, j = t % A.n[1], i = t / A.n[1];
    const double* w = A.coef + 7 * c;
    double s = w[0] * x[c];
    if (i + 1 < A.n[0]) s += w[1] * x[c + sx];
    if (i > 0) s += w[2] * x[c - sx];
    if (j + 1 < A.n[1]) s += w[3] * x[c + sy];
    if (j > 0) s += w[4] * x[c - sy];
    if (k + 1 < A.n[2]) s += w[5] * x[c + 1];
    if (k > 0) s += w[6] * x[c - 1];
    return s;
}

// r = b - A x, rhat = r, p = v = 0; partial sums of r.r and b.b
__global__ void __launch_bounds__(kBlock) bi_start(const __grid_constant__ CoefOp A, int64_t m,
                                                   const double* __restrict__ b, const double* __restrict__ x,
                                                   double* __restrict__ r, double* __restrict__ rhat,
                                                   double* __restrict__ p, double* __restrict__ v,
                                                   double* __restrict__ part, double* __restrict__ part2) {
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double rr = 0.0, bb = 0.0;
    if (c < m) {
        const double rc = b[c] - apply_coef(A, x, c);
        r[c] = rc;
        rhat[c] = rc;
        p[c] = 0.0;
        v[c] = 0.0;
        rr = rc * rc;
        bb = b[c] * b[c];
    }
    block_partial(rr, part);
    __syncthreads();
    block_partial(bb, part2);
}

// p^ = (r + beta (p - omega v)) / d, p holding p^; fresh: rhat = r, p^ = r / d
__global__ void __launch_bounds__(kBlock) bi_direction(const __grid_constant__ CoefOp A, int64_t m,
                                                       const double* __restrict__ r, double* __restrict__ rhat,
                                                       double* __restrict__ p, const double* __restrict__ v,
                                                       const double* __restrict__ S) {
    if (S[bDONE] != 0.0) return;
    const double beta = S[bBETA], omega = S[bOMEGA];
    const bool fresh = S[bFRESH] != 0.0;
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (c >= m) return;
    const double d = row_scale(A.coef[7 * c]), rc = r[c];
    if (fresh) rhat[c] = rc;
    p[c] = (fresh ? rc : rc + beta * (d * p[c] - omega * v[c])) / d;
}

// y = A z; partial sums of a.y (and of y.y when part2 is set)
__global__ void __launch_bounds__(kBlock) bi_apply(const __grid_constant__ CoefOp A, int64_t m,
                                                   const double* __restrict__ z, double* __restrict__ y,
                                                   const double* __restrict__ a, double* __restrict__ part,
                                                   double* __restrict__ part2, const double* __restrict__ S) {
    if (S[bDONE] != 0.0) return;
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double d1 = 0.0, d2 = 0.0;
    if (c < m) {
        const double yc = apply_coef(A, z, c);
        y[c] = yc;
        d1 = a[c] * yc;
        d2 = yc * yc;
    }
    block_partial(d1, part);
    if (part2) {
        __syncthreads();
        block_partial(d2, part2);
    }
}

// s = r - alpha v in r's place, s^ = s / d
__global__ void __launch_bounds__(kBlock) bi_half(const __grid_constant__ CoefOp A, int64_t m, double* __restrict__ r,
                                                  const double* __restrict__ v, double* __restrict__ sv,
                                                  const double* __restrict__ S) {
    if (S[bDONE] != 0.0) return;
    const double alpha = S[bALPHA];
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    if (c >= m) return;
    const double sc = r[c] - alpha * v[c];
    r[c] = sc;
    sv[c] = sc / row_scale(A.coef[7 * c]);
}

// x += alpha p^ + omega s^, r = s - omega t; partial sums of rhat.r and r.r
__global__ void __launch_bounds__(kBlock) bi_update(int64_t m, double* __restrict__ x, double* __restrict__ r,
                                                    const double* __restrict__ rhat, const double* __restrict__ p,
                                                    const double* __restrict__ sv, const double* __restrict__ t,
                                                    double* __restrict__ part, double* __restrict__ part2,
                                                    const double* __restrict__ S) {
    if (S[bDONE] != 0.0) return;
    const double alpha = S[bALPHA], omega = S[bOMEGA];
    const int64_t c = blockIdx.x * (int64_t)kBlock + threadIdx.x;
    double d1 = 0.0, d2 = 0.0;
    if (c < m) {
        x[c] += alpha * p[c] + omega * sv[c];
        const double rc = r[c] - omega * t[c];
        r[c] = rc;
        d1 = rhat[c] * rc;
        d2 = rc * rc;
    }
    block_partial(d1, part);
    __syncthreads();
    block_partial(d2, part2);
}

// One block.  mode 0: start; 1: alpha = rho / rhat.v; 2: omega = t.s / t.t;
// 3: rho', beta, residual and the stopping test, or a fresh start from r.
__global__ void __launch_bounds__(kBlock) bi_scalars(int mode, const double* __restrict__ part,
                                                     const double* __restrict__ part2, int nb, double* S,
                                                     double rel_tol, int64_t max_iter) {
    if (mode != 0 && S[bDONE] != 0.0) return;
    const double a = sum_partials(part, nb);
    __syncthreads();
    const double b = part2 ? sum_partials(part2, nb) : 0.0;
    if (threadIdx.x != 0) return;
    if (mode == 0) {
        S[bRR] = a;
        S[bBB] = b;
        S[bTOL2] = rel_tol * rel_tol * b;
        S[bRHO] = a;          // rhat = r
        S[bRHAT2] = a;
        S[bALPHA] = 1.0;
        S[bOMEGA] = 1.0;
        S[bBETA] = 0.0;
        S[bFRESH] = 1.0;      // first direction p = r
        S[bITERS] = 0.0;
        S[bDONE] = (a <= S[bTOL2] || a == 0.0 || max_iter <= 0) ? 1.0 : 0.0;
    } else if (mode == 1) {
        S[bALPHA] = a != 0.0 ? S[bRHO] / a : 0.0;           // (0: the half step alone, then a fresh start)
    } else if (mode == 2) {
        S[bOMEGA] = b > 0.0 ? a / b : 0.0;                  // a = t.s, b = t.t
    } else {
        S[bITERS] += 1.0;
        S[bRR] = b;
        const double rho = a;
        if (S[bOMEGA] == 0.0 || S[bALPHA] == 0.0 || rho * rho <= kRhoRounding * S[bRHAT2] * b) {
            S[bRHO] = b;
            S[bRHAT2] = b;
            S[bFRESH] = 1.0;
        } else {
            S[bBETA] = (rho / S[bRHO]) * (S[bALPHA] / S[bOMEGA]);
            S[bRHO] = rho;
            S[bFRESH] = 0.0;
        }
        if (b <= S[bTOL2] || b == 0.0 || S[bITERS] >= (double)max_iter) S[bDONE] = 1.0;
    }
}

// ---------------------------------------------------------------------------
// Whole solves in one cooperative kernel.
//
// On a mesh whose vectors fit the SMs' shared memory and registers an
// iteration moves next to nothing; what it costs is launches (5 per CG
// iteration, 8 per BiCGSTAB iteration, replayed as graphs) and the round trips
// of the vectors through L2.  Here each block owns a brick of cells for the
// whole solve, with the vectors of its cells in its shared memory and
// registers; a vector the operator is applied to lies in a brick padded by one
// cell, zeros beyond the box.  A block carries the recurrences of its padding
// cells along (the same FMAs as their owner's, so the same bits), and all that
// passes through global memory is the operator's result on the bricks' faces.
// A grid-wide wait is left where an iteration needs dot products, and those are
// gathered: one wait for CG (Chronopoulos and Gear, J. Comput. Appl. Math. 25,
// 1989: r.r and A r.r together, p.A p by recurrence), two for BiCGSTAB (the sums
// that give rho and |r| are taken with t.s and t.t).  A wait and its sums are
// one step (grid_sums); it is about half of an iteration.  512 threads of 128
// registers: the vectors of up to twelve cells per thread stay resident, and
// latency is covered by cells instead of warps.
// B200, us per iteration, launched form -> this one: CG on 16^3 / 52 x 52 x 54 /
// 64 x 64 x 128 cells 12.5 / 15.2 / 19.4 -> 4.7 / 5.7 / 8.7; BiCGSTAB 20.8 / 28.5 /
// 39.5 -> 11.3 / 14.8 / 27.9 (the launched form's before it had the preconditioner).
// ---------------------------------------------------------------------------
constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxBlocks = 160;
constexpr int kResMaxCg = 12;     // cells per thread: x, A r and A p in registers
constexpr int kResMaxBi = 8;      // r, t, v and x in registers
constexpr int kResMaxSums = 5;
constexpr int kSpinLimit = 1 << 21;   // polls of one wait (~0.5 us each) before the solve gives up
constexpr unsigned long long kGaveUp = ~0ull;   // in place of a wait's number: block 0 gave it up

// A partial sum and the number of the wait it belongs to, written and read as
// one 128-bit access.
struct alignas(16) Slot {
    double value;
    unsigned long long epoch;
};

// The slots of two waits in turn: every block's partial sums, sum by sum, then
// the grid's: slots[(e & 1) * kResMaxSums * (blocks + 1) + ...].
constexpr int kSlotsPerBlock = 4 * kResMaxSums;   // two waits of blocks + 1 slots, for two blocks or more

// What a solve reports: written by block 0 at its end (`finished` stays 0 when
// it left before), and `late` by every block that gave up a wait.
struct ResidentOut {
    double rr, bb, iterations, finished, late;
};

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ void publish(Slot* p, double v, unsigned long long e) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 :: "l"(p), "l"(__double_as_longlong(v)), "l"(e) : "memory");
}

__device__ __forceinline__ unsigned long long poll(const Slot* p, double& v) {
    long long lo;
    unsigned long long e;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(e) : "l"(p) : "memory");
    v = __longlong_as_double(lo);
    return e;
}

struct GridSums {
    double part[8][kResWarps];              // the block's warps
    double all[kResMaxSums];                // the grid's sums
    int late;
};

constexpr int sums_width(int n) { return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : 8; }

// The warp's sums of W = 1, 2, 4 or 8 values, value lane / (32 / W) in each lane:
// while there are several, half the lanes pass half of them on and keep the others.
template <int W>
__device__ __forceinline__ double warp_sums(const double (&a)[W], int lane, int o = 16) {
    if constexpr (W == 1) {
        double v = a[0];
#pragma unroll
        for (; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    } else {
        const bool up = lane & o;
        double half[W / 2];
#pragma unroll
        for (int i = 0; i < W / 2; ++i)
            half[i] = (up ? a[i + W / 2] : a[i]) + __shfl_xor_sync(0xffffffffu, up ? a[i] : a[i + W / 2], o);
        return warp_sums<W / 2>(half, lane, o >> 1);
    }
}

// Wait number e of the grid: each of the N values summed over all threads of
// all blocks, the same bits in every block; everything the blocks wrote before
// the call is visible after it.  False when the wait ran out after `polls` polls:
// then the block leaves its solve and says so in out->late, which is an error of
// the whole solve.  Block 0 passes a wait that it gave up on to every block
// (kGaveUp in place of the sum), so none goes on with a sum of some of them; a
// block that gives up by itself leaves block 0 to give up the next wait.
// Block 0 gathers the partial sums and hands out the grid's,
// each as one 16-byte word with the step's number.  With every block reading
// all partial sums instead, a step among 148 blocks takes 4.1 us for one value,
// 6.3 for two and 7.2 for five, since their polls of the same lines hold up one
// another and the stores they wait for; so it took 3.1 and 3.2 us for one and
// for four without lane 0's fence, which adds 0.1 to 0.4 us to an iteration.
template <int N>
__device__ __forceinline__ bool grid_sums(Slot* slots, ResidentOut* out, int polls, GridSums& G, unsigned long long e,
                                          double (&a)[N]) {
    constexpr int W = sums_width(N);
    constexpr int L = 32 / W;                   // lanes of one value
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double wide[W];
#pragma unroll
    for (int n = 0; n < W; ++n) wide[n] = n < N ? a[n < N ? n : 0] : 0.0;
    double v = warp_sums<W>(wide, lane);
    if (lane % L == 0) G.part[lane / L][warp] = v;
    __syncthreads();
    const int nb = (int)gridDim.x;
    Slot* up = slots + (size_t)(e & 1) * kResMaxSums * (nb + 1);
    Slot* down = up + (size_t)kResMaxSums * nb;
    if (warp == 0) {
        const int n = lane / L, j = lane % L;
        v = 0.0;
#pragma unroll
        for (int i = 0; i < kResWarps; i += L)
            if (i + j < kResWarps) v += G.part[n][i + j];
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (nb == 1) {
            if (j == 0 && n < N) G.all[n] = v;
        } else {
            fence_gpu();          // the block's writes (ordered before this by the barrier) before its words
            if (j == 0 && n < N) publish(up + n * nb + blockIdx.x, v, e);
        }
    }
    if (nb > 1) {
        if (blockIdx.x == 0 && warp >= 1 && warp <= N) {        // warp n + 1 gathers value n
            // a lane's polls are in flight together; past the grid it polls the last block again
            constexpr int kPolls = kResMaxBlocks / 32;
            const Slot* from = up + (warp - 1) * nb;
            double got[kPolls];
            unsigned long long when[kPolls];
            int spins = 0;
            bool all;
            do {
#pragma unroll
                for (int u = 0; u < kPolls; ++u) when[u] = poll(from + min(lane + 32 * u, nb - 1), got[u]);
                all = true;
#pragma unroll
                for (int u = 0; u < kPolls; ++u) all = all && when[u] == e;
            } while (!all && ++spins < polls);
            fence_gpu();          // a lane sees what the blocks whose words it polled wrote before them
            v = 0.0;
#pragma unroll
            for (int u = 0; u < kPolls; ++u) v += lane + 32 * u < nb ? got[u] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const bool whole = __all_sync(0xffffffffu, all);
            // and lane 0 passes it on with the sum: the shuffles order no memory, so the
            // lanes' reads come before its word by the barrier and a fence of its own
            __syncwarp();
            if (lane == 0) {
                fence_gpu();
                publish(down + warp - 1, v, whole ? e : kGaveUp);
            }
        }
        if (warp == 0) {
            if (lane < N) {
                double sum;
                int spins = 0;
                unsigned long long when;
                do when = poll(down + lane, sum);
                while (when != e && when != kGaveUp && ++spins < polls);
                if (when != e) G.late = 1;
                G.all[lane] = sum;
            }
            fence_gpu();          // what the blocks wrote before the wait is read after it
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < N; ++n) a[n] = G.all[n];
    if (G.late == 0) return true;
    if (threadIdx.x == 0) out->late = 1.0;
    return false;
}

// The bricks: b[d] cells along axis d, the last ones fewer; g[d] of them.
struct Bricks {
    int n[3];
    int b[3];
    int g[3];
};

// One brick: its first cell, its cells per axis, and the position of its cells
// in the published vectors (all bricks' cells one after the other, the cells of
// a brick in [i][j][k] order).
struct Brick {
    int o[3];
    int d[3];
    int base;
};

__device__ __forceinline__ Brick brick_at(const Bricks& B, int X, int Y, int Z) {
    Brick k;
    const int at[3] = {X, Y, Z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        k.o[a] = at[a] * B.b[a];
        k.d[a] = min(B.b[a], B.n[a] - k.o[a]);
    }
    k.base = k.o[0] * B.n[1] * B.n[2] + k.d[0] * (k.o[1] * B.n[2] + k.d[1] * k.o[2]);
    return k;
}

// A block's shared arrays: the padded brick, the list of padding cells owned
// by other blocks (their place in the published vectors, and in the padding).
struct Padded {
    double* v;
    int* src;
    unsigned short* dst;
    int halo;          // entries of the list
    int sx, sy;        // strides of the padded brick
    int at;            // padded index of the brick's first cell
};

__host__ __device__ inline int padded_cells(const Bricks& B) { return (B.b[0] + 2) * (B.b[1] + 2) * (B.b[2] + 2); }
__host__ __device__ inline int face_cells(const Bricks& B) {
    return 2 * (B.b[0] * B.b[1] + B.b[1] * B.b[2] + B.b[0] * B.b[2]);
}

// Fill a padded brick with the vector x (in mesh order), zeros beyond the box,
// and list the padding cells that belong to other bricks.  All threads.
__device__ __forceinline__ void open_brick(const Bricks& B, const Brick& K, Padded& P, const double* x, int* count) {
    if (threadIdx.x == 0) *count = 0;
    __syncthreads();
    const int e1 = K.d[1] + 2, e2 = K.d[2] + 2, cells = (K.d[0] + 2) * e1 * e2;
    for (int q = threadIdx.x; q < cells; q += kResThreads) {
        const int k = q % e2, t = q / e2, j = t % e1, i = t / e1;
        const int gi = K.o[0] + i - 1, gj = K.o[1] + j - 1, gk = K.o[2] + k - 1;
        const int out = (i == 0 || i == K.d[0] + 1) + (j == 0 || j == K.d[1] + 1) + (k == 0 || k == K.d[2] + 1);
        const bool box = gi >= 0 && gi < B.n[0] && gj >= 0 && gj < B.n[1] && gk >= 0 && gk < B.n[2];
        const int pad = i * P.sx + j * P.sy + k;
        P.v[pad] = box && out <= 1 ? x[((int64_t)gi * B.n[1] + gj) * B.n[2] + gk] : 0.0;
        if (box && out == 1) {
            const int X = gi / B.b[0], Y = gj / B.b[1], Z = gk / B.b[2];
            const Brick N = brick_at(B, X, Y, Z);
            const int h = atomicAdd(count, 1);
            P.src[h] = N.base + ((gi - N.o[0]) * N.d[1] + (gj - N.o[1])) * N.d[2] + (gk - N.o[2]);
            P.dst[h] = (unsigned short)pad;
        }
    }
    __syncthreads();
    P.halo = *count;
}

// update(entry, padded index, value of pub at the cell's place) for every
// listed padding cell; the loads of four cells in flight.
template <typename Update>
__device__ __forceinline__ void update_halo(const Padded& P, const double* pub, Update update) {
    for (int h = threadIdx.x; h < P.halo; h += 4 * kResThreads) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (h + u * kResThreads < P.halo) v[u] = __ldcg(pub + P.src[h + u * kResThreads]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (h + u * kResThreads < P.halo) update(h + u * kResThreads, P.dst[h + u * kResThreads], v[u]);
    }
}

// Of a thread's cell: its padded index (bits 0..15), kOwned, and kFace when
// another block may read it.  The loops over a thread's cells have no branch on
// kOwned around their arithmetic, so the cells' chains overlap.  (A thread without a
// cell reads the brick's first one, perhaps while its owner writes it: what it makes
// of it goes nowhere.)
constexpr unsigned kOwned = 1u << 16, kFace = 1u << 17;
constexpr unsigned kPlainWarp = 1u << 18;     // bi_resident: its warp's cells all have the plain row

__device__ __forceinline__ unsigned own_cell(const Bricks& B, const Brick& K, const Padded& P, int l, int64_t* c) {
    const int k = l % K.d[2], t = l / K.d[2], j = t % K.d[1], i = t / K.d[1];
    *c = ((int64_t)(K.o[0] + i) * B.n[1] + K.o[1] + j) * B.n[2] + K.o[2] + k;
    const bool face = i == 0 || i == K.d[0] - 1 || j == 0 || j == K.d[1] - 1 || k == 0 || k == K.d[2] - 1;
    return (unsigned)(P.at + i * P.sx + j * P.sy + k) | kOwned | (face ? kFace : 0u);
}

// diag x + the six couplings, in the order of the reference's rows
// (+x -x +y -y +z -z; zeros beyond the box).
__device__ __forceinline__ double apply_padded(double diag, const double w[6], const double* x, int at, int sx, int sy) {
    double s = diag * x[at];
    s = fma(w[0], x[at + sx], s);
    s = fma(w[1], x[at - sx], s);
    s = fma(w[2], x[at + sy], s);
    s = fma(w[3], x[at - sy], s);
    s = fma(w[4], x[at + 1], s);
    return fma(w[5], x[at - 1], s);
}

// The kernels' common start: the block's brick and its shared arrays.
__device__ __forceinline__ Brick start_brick(const Bricks& B, double* shared, Padded& P) {
    const int Z = (int)blockIdx.x % B.g[2], t = (int)blockIdx.x / B.g[2];
    P.v = shared;
    P.sy = B.b[2] + 2;
    P.sx = (B.b[1] + 2) * P.sy;
    P.at = P.sx + P.sy + 1;
    return brick_at(B, t / B.g[1], t % B.g[1], Z);
}

// Conjugate gradients.  Thread t owns the brick's cells t, t + 512, ... (at most
// S): x, w = A r and q = A p in registers, p in shared memory, r in the padded
// brick, and of the padding cells r there and q in a list.  With rr = r.r,
// beta = rr / rr_old and alpha = rr / (w.r - beta rr / alpha_old) (p.A p by
// recurrence): p = r + beta p, q = w + beta q, x += alpha p, r -= alpha q.  The
// stopping test is that of the launched form.
template <int S>
__global__ void __launch_bounds__(kResThreads, 1)
    cg_resident(const __grid_constant__ PoissonOp A, const __grid_constant__ Bricks B, const double* __restrict__ rhs,
                double* x_out, double* w_pub, int64_t m, Slot* slots, ResidentOut* out, double rel_tol,
                int64_t max_iter, int polls) {
    extern __shared__ double shared[];
    __shared__ GridSums G;
    __shared__ int count;
    Padded P;
    const Brick K = start_brick(B, shared, P);
    double* r = P.v;
    double* p = shared + padded_cells(B);
    double* halo_q = p + S * kResThreads;
    P.src = reinterpret_cast<int*>(halo_q + face_cells(B));
    P.dst = reinterpret_cast<unsigned short*>(P.src + face_cells(B));
    if (threadIdx.x == 0) G.late = 0;
    open_brick(B, K, P, x_out, &count);
    const int cells = K.d[0] * K.d[1] * K.d[2];
    const double off[6] = {A.off[0], A.off[0], A.off[1], A.off[1], A.off[2], A.off[2]};
    double x[S], w[S], q[S];
    unsigned own[S];
    double first[2] = {0.0, 0.0};                  // r.r and b.b
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int l = threadIdx.x + s * kResThreads;
        x[s] = w[s] = q[s] = 0.0;
        p[l] = 0.0;
        own[s] = P.at;             // past the brick's cells: its first one, read and never written
        if (l < cells) {
            int64_t c;
            own[s] = own_cell(B, K, P, l, &c);
            const int at = own[s] & 0xffff;
            x[s] = r[at];
            const double bc = rhs[c];
            w[s] = bc - apply_padded(A.diag, off, r, at, P.sx, P.sy);
            if (own[s] & kFace) w_pub[m + K.base + l] = w[s];
            first[0] = fma(w[s], w[s], first[0]);
            first[1] = fma(bc, bc, first[1]);
        }
    }
    for (int h = threadIdx.x; h < P.halo; h += kResThreads) halo_q[h] = 0.0;
    unsigned long long epoch = 1;
    if (!grid_sums(slots, out, polls, G, epoch, first)) return;
#pragma unroll
    for (int s = 0; s < S; ++s)                    // the padded brick held x; now r
        if (own[s] & kOwned) r[own[s] & 0xffff] = w[s];
    update_halo(P, w_pub + m, [&](int, int at, double rc) { r[at] = rc; });
    const double bb = first[1], tol2 = rel_tol * rel_tol * bb;
    double rr = first[0], rr_old = 0.0, alpha = 0.0;
    int64_t it = 0;
    bool done = rr <= tol2 || rr == 0.0 || max_iter <= 0;
    while (!done) {
        __syncthreads();
        // two buffers: a block may be one wait ahead of another's reading
        double* pub = w_pub + (it & 1) * m;
        double sum[2] = {0.0, 0.0};                // r.r and w.r
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int at = own[s] & 0xffff;
            const bool mine = own[s] & kOwned;
            w[s] = apply_padded(A.diag, off, r, at, P.sx, P.sy);
            const double rc = mine ? r[at] : 0.0;
            if (own[s] & kFace) pub[K.base + threadIdx.x + s * kResThreads] = w[s];
            sum[0] = fma(rc, rc, sum[0]);
            sum[1] = fma(w[s], rc, sum[1]);
        }
        if (!grid_sums(slots, out, polls, G, ++epoch, sum)) return;
        rr = sum[0];
        if (rr <= tol2 || rr == 0.0 || it >= max_iter) break;
        const double beta = it == 0 ? 0.0 : rr / rr_old;
        alpha = rr / (it == 0 ? sum[1] : sum[1] - beta * rr / alpha);
        rr_old = rr;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int l = threadIdx.x + s * kResThreads, at = own[s] & 0xffff;
            const double rc = r[at], pc = fma(beta, p[l], rc);
            p[l] = pc;
            q[s] = fma(beta, q[s], w[s]);
            x[s] = fma(alpha, pc, x[s]);
            if (own[s] & kOwned) r[at] = fma(-alpha, q[s], rc);
        }
        update_halo(P, pub, [&](int h, int at, double wc) {
            const double qc = fma(beta, halo_q[h], wc);
            halo_q[h] = qc;
            r[at] = fma(-alpha, qc, r[at]);
        });
        ++it;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (own[s] & kOwned) {
            int64_t c;
            own_cell(B, K, P, threadIdx.x + s * kResThreads, &c);
            x_out[c] = x[s];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out->rr = rr;
        out->bb = bb;
        out->iterations = (double)it;
        out->finished = 1.0;
    }
}

// What a cell's coefficient row is, decided once per solve: most rows are the
// plain Laplacian's (the couplings in bits 0..5 present, the others zero) or a
// conductor's identity, and need no load; the others are read from coef.
constexpr unsigned kRowIdentity = 64u, kRowStored = 128u;

__device__ __forceinline__ unsigned classify_row(const PoissonOp& A, const double* __restrict__ w) {
    unsigned mask = 0;
    bool plain = true;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const double v = w[1 + d];
        if (v != 0.0) mask |= 1u << d;
        plain = plain && (v == 0.0 || v == A.off[d >> 1]);
    }
    if (plain && w[0] == A.diag) return mask;
    if (w[0] == 1.0 && mask == 0u) return kRowIdentity;
    return kRowStored;
}

// Rows in shared memory: the plain ones by their mask of couplings (0..63), the
// identity (64), and the stored rows of the brick's cells as far as they fit
// (about 300 of its 4000 cells lie next to a conductor's surface); the others
// are read from coef at every use.
struct Row {
    double w[7];
    double scale;    // what the preconditioner divides by, and its reciprocal
    double inv;      // (nine doubles: an odd stride, so the lanes' rows lie in all banks)
};
constexpr int kFixedRows = 65;

__device__ __forceinline__ double apply_row(const double* row, const double* x, int at, int sx, int sy) {
    const double w[6] = {row[1], row[2], row[3], row[4], row[5], row[6]};
    return apply_padded(row[0], w, x, at, sx, sy);
}

constexpr double kSumRounding = 1e-10;     // of s.s: r.r = s.s - 2 omega t.s + omega^2 t.t to 1e-5 above it

// BiCGSTAB over per-cell rows (preconditioned and restarted as the launched form).
// p^ and s^ in padded bricks, x and rhat in shared memory, r (then s), t, v and x in
// registers; p = d p^; of the padding cells r, v and d in lists.  rho = rhat.r and
// r.r come from the sums taken with t: r = s - omega t.  A warp whose 32 cells all
// have the plain row takes its constants; another reads rows.
template <int S>
__global__ void __launch_bounds__(kResThreads, 1)
    bi_resident(const __grid_constant__ PoissonOp A, const __grid_constant__ Bricks B,
                const double* __restrict__ coef, const double* __restrict__ rhs, double* x_out, double* v_pub,
                double* t_pub, int row_space, Slot* slots, ResidentOut* out, double rel_tol, int64_t max_iter, int polls) {
    extern __shared__ double shared[];
    __shared__ GridSums G;
    __shared__ int count, n_rows;
    Padded P;
    const Brick K = start_brick(B, shared, P);
    const int pads = padded_cells(B), faces = face_cells(B);
    double* p = P.v;
    double* half = shared + pads;
    double* rhat = half + pads;
    double* halo_r = rhat + S * kResThreads;
    double* halo_v = halo_r + faces;
    double* halo_diag = halo_v + faces;
    double* halo_inv = halo_diag + faces;
    Row* rows = reinterpret_cast<Row*>(halo_inv + faces);
    P.src = reinterpret_cast<int*>(rows + row_space);
    P.dst = reinterpret_cast<unsigned short*>(P.src + faces);
    const double inv_plain = 1.0 / A.diag;
    if (threadIdx.x == 0) {
        G.late = 0;
        n_rows = kFixedRows;
    }
    for (int q = threadIdx.x; q < kFixedRows; q += kResThreads) {
        rows[q].w[0] = q == 64 ? 1.0 : A.diag;
        rows[q].scale = rows[q].w[0];
        rows[q].inv = q == 64 ? 1.0 : inv_plain;
        for (int d = 0; d < 6; ++d) rows[q].w[1 + d] = q < 64 && (q & (1 << d)) ? A.off[d >> 1] : 0.0;
    }
    for (int q = threadIdx.x; q < pads; q += kResThreads) half[q] = 0.0;
    open_brick(B, K, P, x_out, &count);
    // the diagonals of the padding cells, by their place in the padded brick
    for (int h = threadIdx.x; h < P.halo; h += kResThreads) {
        const int pad = P.dst[h], i = pad / P.sx, j = (pad - i * P.sx) / P.sy, k = pad - i * P.sx - j * P.sy;
        const int64_t c = ((int64_t)(K.o[0] + i - 1) * B.n[1] + K.o[1] + j - 1) * B.n[2] + K.o[2] + k - 1;
        halo_diag[h] = row_scale(coef[7 * c]);
        halo_inv[h] = halo_diag[h] == A.diag ? inv_plain : 1.0 / halo_diag[h];
        halo_v[h] = 0.0;
    }
    const int cells = K.d[0] * K.d[1] * K.d[2];
    const double off[6] = {A.off[0], A.off[0], A.off[1], A.off[1], A.off[2], A.off[2]};
    double r[S], t[S], v[S], x[S];
    unsigned own[S];
    int row[S];                // of its cell: the row in shared memory, or -1 - cell: in coef
    double first[2] = {0.0, 0.0};                  // r.r and b.b
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int l = threadIdx.x + s * kResThreads;
        r[s] = t[s] = v[s] = x[s] = 0.0;
        rhat[l] = 0.0;
        own[s] = P.at;             // past the brick's cells: its first one, read and never written
        row[s] = 63;
        if (l < cells) {
            int64_t c;
            own[s] = own_cell(B, K, P, l, &c);
            const double* mine = coef + 7 * c;
            const unsigned kind = classify_row(A, mine);
            row[s] = (int)kind;
            if (kind & kRowStored) {
                row[s] = -1 - (int)c;
                const int n = atomicAdd(&n_rows, 1);
                if (n < row_space) {
#pragma unroll
                    for (int d = 0; d < 7; ++d) rows[n].w[d] = mine[d];
                    rows[n].scale = row_scale(mine[0]);
                    rows[n].inv = rows[n].scale == A.diag ? inv_plain : 1.0 / rows[n].scale;
                    row[s] = n;
                }
            }
            const int at = own[s] & 0xffff;
            x[s] = p[at];
            const double bc = rhs[c];
            r[s] = bc - apply_row(mine, p, at, P.sx, P.sy);
            rhat[l] = r[s];
            if (own[s] & kFace) t_pub[K.base + l] = r[s];
            first[0] = fma(r[s], r[s], first[0]);
            first[1] = fma(bc, bc, first[1]);
        }
        // (the past-the-end cells of a warp count as plain: nothing of theirs is kept)
        if (__all_sync(0xffffffffu, row[s] == 63)) own[s] |= kPlainWarp;
    }
    unsigned long long epoch = 1;
    if (!grid_sums(slots, out, polls, G, epoch, first)) return;
    update_halo(P, t_pub, [&](int h, int, double rc) { halo_r[h] = rc; });
    double rr = first[0], rho = rr, beta = 0.0, omega = 1.0;
    double rhat2 = rr;                 // |rhat|^2
    bool fresh = true;                 // p = r: the first direction, and after a restart
    bool restart = false;
    const double bb = first[1], tol2 = rel_tol * rel_tol * bb;
    int64_t it = 0;
    bool done = rr <= tol2 || rr == 0.0 || max_iter <= 0;
    // formed alike for a cell and for its copies in other bricks' padding
    auto direction = [&](double d, double ph, double vc, double rc) {
        return fresh ? rc : fma(beta, fma(-omega, vc, d * ph), rc);
    };
    auto own_diag = [&](int s, double& d, double& inv) {
        d = A.diag;
        inv = inv_plain;
        if (!(own[s] & kPlainWarp)) {
            if (row[s] >= 0) {
                d = rows[row[s]].scale;
                inv = rows[row[s]].inv;
            } else {
                d = row_scale(coef[7 * (int64_t)(-1 - row[s])]);
                inv = d == A.diag ? inv_plain : 1.0 / d;
            }
        }
    };
    auto apply = [&](int s, const double* vec) {
        const int at = own[s] & 0xffff;
        if (own[s] & kPlainWarp) return apply_padded(A.diag, off, vec, at, P.sx, P.sy);
        return apply_row(row[s] >= 0 ? rows[row[s]].w : coef + 7 * (int64_t)(-1 - row[s]), vec, at, P.sx, P.sy);
    };
    while (!done) {
        if (restart) {
            // rhat = r: the old one has nothing left to say about r
            double sum[1] = {0.0};
#pragma unroll
            for (int s = 0; s < S; ++s) {
                rhat[threadIdx.x + s * kResThreads] = r[s];
                sum[0] = fma(r[s], r[s], sum[0]);
            }
            if (!grid_sums(slots, out, polls, G, ++epoch, sum)) return;
            rr = rho = rhat2 = sum[0];
            if (rr <= tol2 || rr == 0.0) break;
            fresh = true;
            restart = false;
        }
        // p^ = (r + beta (p - omega v)) / d, v = A p^
        for (int h = threadIdx.x; h < P.halo; h += kResThreads) {
            const int at = P.dst[h];
            p[at] = halo_inv[h] * direction(halo_diag[h], p[at], halo_v[h], halo_r[h]);
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int at = own[s] & 0xffff;
            double d, inv;
            own_diag(s, d, inv);
            const double ph = inv * direction(d, p[at], v[s], r[s]);
            if (own[s] & kOwned) p[at] = ph;
        }
        fresh = false;
        __syncthreads();
        double dv[1] = {0.0};
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int l = threadIdx.x + s * kResThreads;
            v[s] = apply(s, p);
            if (own[s] & kFace) v_pub[K.base + l] = v[s];
            dv[0] = fma(rhat[l], v[s], dv[0]);           // rhat is zero past the brick's cells
        }
        if (!grid_sums(slots, out, polls, G, ++epoch, dv)) return;
        if (dv[0] == 0.0) {
            restart = true;
            done = ++it >= max_iter;
            continue;
        }
        const double alpha = rho / dv[0];
        // s = r - alpha v, t = A (s / d)
        update_halo(P, v_pub, [&](int h, int at, double vc) {
            halo_v[h] = vc;
            const double sc = fma(-alpha, vc, halo_r[h]);
            halo_r[h] = sc;
            half[at] = halo_inv[h] * sc;
        });
#pragma unroll
        for (int s = 0; s < S; ++s) {
            double d, inv;
            own_diag(s, d, inv);
            r[s] = own[s] & kOwned ? fma(-alpha, v[s], r[s]) : 0.0;
            if (own[s] & kOwned) half[own[s] & 0xffff] = inv * r[s];
        }
        __syncthreads();
        double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};               // t.s, t.t, rhat.s, rhat.t, s.s
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int l = threadIdx.x + s * kResThreads;
            const double tc = apply(s, half);
            t[s] = own[s] & kOwned ? tc : 0.0;
            if (own[s] & kFace) t_pub[K.base + l] = tc;
            sum[0] = fma(r[s], t[s], sum[0]);
            sum[1] = fma(t[s], t[s], sum[1]);
            sum[2] = fma(rhat[l], r[s], sum[2]);
            sum[3] = fma(rhat[l], t[s], sum[3]);
            sum[4] = fma(r[s], r[s], sum[4]);
        }
        if (!grid_sums(slots, out, polls, G, ++epoch, sum)) return;
        omega = sum[1] > 0.0 ? sum[0] / sum[1] : 0.0;
        // x += alpha p^ + omega s^, r = s - omega t
        update_halo(P, t_pub, [&](int h, int, double tc) { halo_r[h] = fma(-omega, tc, halo_r[h]); });
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int at = own[s] & 0xffff;
            x[s] += fma(alpha, p[at], omega * half[at]);         // (past the brick's cells: never stored)
            r[s] = fma(-omega, t[s], r[s]);
        }
        ++it;
        rr = fma(omega, fma(omega, sum[1], -2.0 * sum[0]), sum[4]);
        // (rhat.s vanishes but for rounding: without it rho would drift from rhat.r)
        const double rho_new = fma(-omega, sum[3], sum[2]);
        beta = omega != 0.0 ? (rho_new / rho) * (alpha / omega) : 0.0;
        rho = rho_new;
        // near zero that is the rounding of its terms: before the solve ends on it, or the
        // next step starts from it, r.r itself
        if (rr <= tol2 || rr <= kSumRounding * sum[4] || it >= max_iter) {
            double own_rr[1] = {0.0};
#pragma unroll
            for (int s = 0; s < S; ++s) own_rr[0] = fma(r[s], r[s], own_rr[0]);
            if (!grid_sums(slots, out, polls, G, ++epoch, own_rr)) return;
            rr = own_rr[0];
        }
        done = rr <= tol2 || rr == 0.0 || it >= max_iter;
        // rhat.r is rounding alone (rhat lives on the cells with charge, r elsewhere by now)
        restart = omega == 0.0 || rho * rho <= kRhoRounding * rhat2 * rr;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (own[s] & kOwned) {
            int64_t c;
            own_cell(B, K, P, threadIdx.x + s * kResThreads, &c);
            x_out[c] = x[s];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out->rr = rr;
        out->bb = bb;
        out->iterations = (double)it;
        out->finished = 1.0;
    }
}

// The bricks of a resident solve, its cells per thread (0: the mesh does not
// fit) and its shared memory.  One block on each SM at most, and one per 1024
// cells, rounded up to 256 (two from 1793 cells): a wait costs less among few blocks.  Of the ways to cut the mesh: the
// one with the fewest cells and padding cells per brick.
struct ResidentPlan {
    Bricks bricks;
    int per_thread;
    int blocks;
    size_t smem;
    Slot* slots;
    ResidentOut* out;
    int polls;         // of a grid-wide wait, at most
};

constexpr size_t kResSharedLimit = 224 * 1024;   // with the static arrays below the 227 KB of a block

static cudaError_t plan_resident(const int64_t n[3], int most, int padded_vectors, int plain_vectors,
                                 int face_vectors, double* spare, double* sums, int polls, ResidentPlan* plan) {
    plan->per_thread = 0;
    int dev = 0, sms = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (e != cudaSuccess || !coop) return e;
    const int64_t m = n[0] * n[1] * n[2];
    if (m > (int64_t)kResMaxBlocks * most * kResThreads) return cudaSuccess;
    int64_t top = (m + kBlock - 1) / kBlock / 4;
    if (top > sms) top = sms;
    if (top > kResMaxBlocks) top = kResMaxBlocks;
    if (top < 1) top = 1;
    int64_t best = -1;
    for (int64_t gx = 1; gx <= top && gx <= n[0]; ++gx)
        for (int64_t gy = 1; gx * gy <= top && gy <= n[1]; ++gy) {
            const int64_t gz = top / (gx * gy) < n[2] ? top / (gx * gy) : n[2];
            const int64_t bx = (n[0] + gx - 1) / gx, by = (n[1] + gy - 1) / gy, bz = (n[2] + gz - 1) / gz;
            const int64_t cells = bx * by * bz, faces = 2 * (bx * by + by * bz + bx * bz);
            const int64_t pads = (bx + 2) * (by + 2) * (bz + 2);
            if (cells > (int64_t)most * kResThreads || pads > 0xffff) continue;
            int s = 1;
            while (s * kResThreads < cells) s = s < 8 ? 2 * s : 12;
            const size_t smem = sizeof(double) * ((size_t)padded_vectors * pads + (size_t)plain_vectors * s * kResThreads) +
                                (size_t)faces * (face_vectors * sizeof(double) + sizeof(int) + sizeof(unsigned short));
            const int64_t cost = cells + faces;
            if (smem + kFixedRows * sizeof(Row) > kResSharedLimit || (best >= 0 && cost >= best)) continue;
            best = cost;
            plan->per_thread = s;
            plan->smem = smem;
            const int64_t b[3] = {bx, by, bz};
            plan->blocks = 1;
            for (int a = 0; a < 3; ++a) {
                plan->bricks.n[a] = (int)n[a];
                plan->bricks.b[a] = (int)b[a];
                plan->bricks.g[a] = (int)((n[a] + b[a] - 1) / b[a]);
                plan->blocks *= plan->bricks.g[a];
            }
        }
    // The slots lie in a vector of the scratch that the resident form leaves free
    // (896 cells and more for each block's 320 bytes; none for a single block);
    // a caller's scratch is aligned for doubles, the slots need 16 bytes.  The
    // report goes where the launched form keeps its sums.
    static_assert(kSlotsPerBlock * sizeof(Slot) + 8 <= 896 * sizeof(double), "a block's slots fit its cells' scratch");
    static_assert(sizeof(ResidentOut) <= 9 * sizeof(double), "the report fits the sums' scratch");
    plan->slots = reinterpret_cast<Slot*>((reinterpret_cast<uintptr_t>(spare) + 15) & ~(uintptr_t)15);
    plan->out = reinterpret_cast<ResidentOut*>(sums);
    plan->polls = polls;
    return cudaSuccess;
}

// In place of a status: the device did not take the cooperative launch (its blocks
// would not all be resident: SMs held by another partition or process), and
// nothing of the solve has run.
constexpr int kNotLaunched = 1;

// Launch a resident kernel and read its report back (synchronises s).
static int run_resident(const void* kernel, const ResidentPlan& plan, void** args, int64_t* iterations,
                        double* rel_residual, cudaStream_t s) {
    // always the same limit: it belongs to the kernel, and another thread may be
    // between its own setting and its launch
    PPT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSharedLimit));
    PPT_CUDA_TRY(cudaMemsetAsync(plan.out, 0, sizeof(ResidentOut), s));
    if (plan.blocks > 1)
        PPT_CUDA_TRY(cudaMemsetAsync(plan.slots, 0, (size_t)plan.blocks * kSlotsPerBlock * sizeof(Slot), s));
    const cudaError_t launched =
        plan.polls > 0 ? cudaLaunchCooperativeKernel(kernel, dim3(plan.blocks), dim3(kResThreads), args, plan.smem, s)
                       : cudaErrorCooperativeLaunchTooLarge;     // (a test's refusal)
    if (launched != cudaSuccess) {
        cudaGetLastError();          // an error of the context shows again in the launched form
        return kNotLaunched;
    }
    ResidentOut host;
    PPT_CUDA_TRY(cudaMemcpyAsync(&host, plan.out, sizeof(host), cudaMemcpyDeviceToHost, s));
    PPT_CUDA_TRY(cudaStreamSynchronize(s));
    if (host.finished != 1.0 || host.late != 0.0) return fail(PPT_ERR_TIMEOUT, "a grid-wide wait of the solver ran out");
    if (iterations) *iterations = (int64_t)host.iterations;
    if (rel_residual) *rel_residual = host.bb > 0.0 ? std::sqrt(host.rr / host.bb) : 0.0;
    return PPT_OK;
}

// Iterations of a solve that the resident kernels do not take (a larger mesh, or a
// refused launch): kIterPerGraph of them captured once as a CUDA graph on a private
// stream (the caller's may be the legacy default stream, which cannot be captured)
// and replayed until the device-side stop flag is set; one host check per replay.  The kernels and their order are those of plain
// launches, so the results are the same bits, with a fraction of the launch
// cost (a solve is thousands of short launches on L2-resident vectors).
constexpr int kIterPerGraph = 16;

template <typename Enqueue>
static int run_iterations(cudaStream_t caller, const double* S, int done_slot, int n_scalars, int64_t max_iter,
                          double* host, Enqueue enqueue_iteration) {
    cudaStream_t side = nullptr;
    cudaEvent_t ready = nullptr, finished = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&finished, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(ready, caller);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side, ready, 0);
    if (e == cudaSuccess) e = cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        for (int it = 0; it < kIterPerGraph; ++it) enqueue_iteration(side);
        e = cudaStreamEndCapture(side, &graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    for (int64_t done = 0; e == cudaSuccess;) {
        e = cudaGraphLaunch(exec, side);
        if (e == cudaSuccess) e = cudaMemcpyAsync(host, S, n_scalars * sizeof(double), cudaMemcpyDeviceToHost, side);
        if (e == cudaSuccess) e = cudaStreamSynchronize(side);
        done += kIterPerGraph;
        if (e != cudaSuccess || host[done_slot] != 0.0 || done >= max_iter) break;
    }
    // the caller's stream continues after the solve
    if (e == cudaSuccess) e = cudaEventRecord(finished, side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(caller, finished, 0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (ready) cudaEventDestroy(ready);
    if (finished) cudaEventDestroy(finished);
    if (side) cudaStreamDestroy(side);
    if (e != cudaSuccess) return cuda_fail(e, "solver iterations");
    return PPT_OK;
}

static int mesh_geom(const ppt_mesh_desc* mesh, int64_t n[3], double h[3]) {
    if (!mesh) return fail(PPT_ERR_ARG, "mesh must not be NULL");
    int64_t total = 1;
    for (int a = 0; a < 3; ++a) {
        if (mesh->cells[a] < 1) return fail(PPT_ERR_ARG, "every mesh axis needs at least 1 cell");
        if (!(mesh->extent[a] > 0.0)) return fail(PPT_ERR_ARG, "mesh extents must be positive");
        n[a] = mesh->cells[a];
        h[a] = mesh->extent[a] / (double)mesh->cells[a];
        total *= n[a];
        if (total > (1LL << 34)) return fail(PPT_ERR_ARG, "mesh too large");
    }
    return PPT_OK;
}

// The rows of cells away from conductors.
static PoissonOp laplacian(const int64_t n[3], const double h[3]) {
    PoissonOp A;
    A.diag = 0.0;
    for (int a = 0; a < 3; ++a) {
        A.n[a] = n[a];
        A.off[a] = -2.0 / (h[a] * (h[a] + h[a]));
        A.diag += 2.0 / (h[a] * h[a]);
    }
    return A;
}

}  // namespace ppt

using namespace ppt;

extern "C" int64_t ppt_poisson_scratch_bytes(const ppt_mesh_desc* mesh) {
    int64_t n[3];
    double h[3];
    if (mesh_geom(mesh, n, h)) return -1;
    const int64_t m = n[0] * n[1] * n[2];
    const int64_t nb = (m + kBlock - 1) / kBlock;
    return (3 * m + 2 * nb + kNumScalars) * (int64_t)sizeof(double);
}

static int solve_laplacian(const ppt_mesh_desc* mesh, const double* rhs, double* phi, void* scratch, double rel_tol,
                           int64_t max_iter, int polls, int64_t* iterations, double* rel_residual, void* stream) {
    int64_t n[3];
    double h[3];
    int rc = mesh_geom(mesh, n, h);
    if (rc) return rc;
    if (!rhs || !phi || !scratch) return fail(PPT_ERR_ARG, "rhs, phi and scratch must not be NULL");
    if (!(rel_tol >= 0.0)) return fail(PPT_ERR_ARG, "rel_tol must be >= 0");
    PoissonOp A = laplacian(n, h);
    const int64_t m = n[0] * n[1] * n[2];
    const int nb = (int)((m + kBlock - 1) / kBlock);
    double* r = static_cast<double*>(scratch);
    double* p = r + m;
    double* q = p + m;
    double* part = q + m;
    double* part2 = part + nb;
    double* S = part2 + nb;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double host[kNumScalars];
    ResidentPlan plan;
    PPT_CUDA_TRY(plan_resident(n, kResMaxCg, 1, 1, 1, q, part, polls, &plan));
    if (plan.per_thread) {
        int64_t mm = m;
        double* w_pub = r;            // two buffers; q is left for the slots
        void* args[] = {&A,   &plan.bricks, &rhs,      &phi,      &w_pub,
                        &mm,  &plan.slots,  &plan.out, &rel_tol,  &max_iter, &plan.polls};
        const void* kernel = plan.per_thread == 1   ? (const void*)cg_resident<1>
                             : plan.per_thread == 2 ? (const void*)cg_resident<2>
                             : plan.per_thread == 4 ? (const void*)cg_resident<4>
                             : plan.per_thread == 8 ? (const void*)cg_resident<8>
                                                    : (const void*)cg_resident<12>;
        rc = run_resident(kernel, plan, args, iterations, rel_residual, s);
        if (rc != kNotLaunched) return rc;
    }
    cg_start<<<nb, kBlock, 0, s>>>(A, m, rhs, phi, r, p, part, part2);
    cg_scalars<<<1, kBlock, 0, s>>>(0, part, part2, nb, S, rel_tol, max_iter);
    PPT_CUDA_TRY(cudaGetLastError());
    // Graph replays of kIterPerGraph iterations between host checks; a
    // finished solve turns the remaining launches of a replay into no-ops.
    rc = run_iterations(s, S, kDONE, kNumScalars, max_iter, host, [&](cudaStream_t st) {
        cg_apply<<<nb, kBlock, 0, st>>>(A, m, p, q, part, S);
        cg_scalars<<<1, kBlock, 0, st>>>(1, part, nullptr, nb, S, rel_tol, max_iter);
        cg_step<<<nb, kBlock, 0, st>>>(m, phi, r, p, q, part, S);
        cg_scalars<<<1, kBlock, 0, st>>>(2, part, nullptr, nb, S, rel_tol, max_iter);
        cg_direction<<<nb, kBlock, 0, st>>>(m, r, p, S);
    });
    if (rc) return rc;
    if (iterations) *iterations = (int64_t)host[kITERS];
    if (rel_residual) *rel_residual = host[kBB] > 0.0 ? std::sqrt(host[kRR] / host[kBB]) : 0.0;
    return PPT_OK;
}

extern "C" int ppt_poisson_solve(const ppt_mesh_desc* mesh, const double* rhs, double* phi, void* scratch,
                                 double rel_tol, int64_t max_iter, int64_t* iterations, double* rel_residual,
                                 void* stream) {
    return solve_laplacian(mesh, rhs, phi, scratch, rel_tol, max_iter, kSpinLimit, iterations, rel_residual, stream);
}

extern "C" int ppt_field_from_potential(const ppt_mesh_desc* mesh, const double* phi, double* ex, double* ey,
                                        double* ez, void* stream) {
    int64_t n[3];
    double h[3];
    int rc = mesh_geom(mesh, n, h);
    if (rc) return rc;
    if (!phi) return fail(PPT_ERR_ARG, "phi must not be NULL");
    const int64_t m = n[0] * n[1] * n[2];
    field_from_potential<<<(unsigned)((m + kBlock - 1) / kBlock), kBlock, 0, static_cast<cudaStream_t>(stream)>>>(
        n[0], n[1], n[2], phi, h[0], h[1], h[2], ex, ey, ez);
    PPT_CUDA_TRY(cudaGetLastError());
    return PPT_OK;
}

extern "C" int64_t ppt_poisson_coef_scratch_bytes(const ppt_mesh_desc* mesh) {
    int64_t n[3];
    double h[3];
    if (mesh_geom(mesh, n, h)) return -1;
    const int64_t m = n[0] * n[1] * n[2];
    const int64_t nb = (m + kBlock - 1) / kBlock;
    return (6 * m + 2 * nb + bNumScalars) * (int64_t)sizeof(double);
}

static int solve_coef(const ppt_mesh_desc* mesh, const double* coef, const double* rhs, double* phi, void* scratch,
                      double rel_tol, int64_t max_iter, int polls, int64_t* iterations, double* rel_residual,
                      void* stream) {
    int64_t n[3];
    double h[3];
    int rc = mesh_geom(mesh, n, h);
    if (rc) return rc;
    if (!coef || !rhs || !phi || !scratch) return fail(PPT_ERR_ARG, "coef, rhs, phi and scratch must not be NULL");
    if (!(rel_tol >= 0.0)) return fail(PPT_ERR_ARG, "rel_tol must be >= 0");
    CoefOp A;
    for (int a = 0; a < 3; ++a) A.n[a] = n[a];
    A.coef = coef;
    const int64_t m = n[0] * n[1] * n[2];
    const int nb = (int)((m + kBlock - 1) / kBlock);
    double* r = static_cast<double*>(scratch);
    double* rhat = r + m;
    double* p = rhat + m;
    double* v = p + m;
    double* sv = v + m;
    double* t = sv + m;
    double* part = t + m;
    double* part2 = part + nb;
    double* S = part2 + nb;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double host[bNumScalars];
    ResidentPlan plan;
    PPT_CUDA_TRY(plan_resident(n, kResMaxBi, 2, 1, 4, p, part, polls, &plan));
    if (plan.per_thread) {
        PoissonOp L = laplacian(n, h);
        double* v_pub = r;
        double* t_pub = rhat;
        // what is left of the shared memory holds coefficient rows
        int row_space = (int)((kResSharedLimit - plan.smem) / sizeof(Row));
        if (row_space > plan.per_thread * kResThreads + kFixedRows) row_space = plan.per_thread * kResThreads + kFixedRows;
        plan.smem += (size_t)row_space * sizeof(Row);
        void* args[] = {&L,         &plan.bricks, &coef,     &rhs,     &phi,      &v_pub,     &t_pub, &row_space,
                        &plan.slots, &plan.out,   &rel_tol, &max_iter, &plan.polls};
        const void* kernel = plan.per_thread == 1   ? (const void*)bi_resident<1>
                             : plan.per_thread == 2 ? (const void*)bi_resident<2>
                             : plan.per_thread == 4 ? (const void*)bi_resident<4>
                                                    : (const void*)bi_resident<8>;
        rc = run_resident(kernel, plan, args, iterations, rel_residual, st);
        if (rc != kNotLaunched) return rc;
    }
    bi_start<<<nb, kBlock, 0, st>>>(A, m, rhs, phi, r, rhat, p, v, part, part2);
    bi_scalars<<<1, kBlock, 0, st>>>(0, part, part2, nb, S, rel_tol, max_iter);
    PPT_CUDA_TRY(cudaGetLastError());
    rc = run_iterations(st, S, bDONE, bNumScalars, max_iter, host, [&](cudaStream_t ss) {
        bi_direction<<<nb, kBlock, 0, ss>>>(A, m, r, rhat, p, v, S);
        bi_apply<<<nb, kBlock, 0, ss>>>(A, m, p, v, rhat, part, nullptr, S);
        bi_scalars<<<1, kBlock, 0, ss>>>(1, part, nullptr, nb, S, rel_tol, max_iter);
        bi_half<<<nb, kBlock, 0, ss>>>(A, m, r, v, sv, S);
        bi_apply<<<nb, kBlock, 0, ss>>>(A, m, sv, t, r, part, part2, S);
        bi_scalars<<<1, kBlock, 0, ss>>>(2, part, part2, nb, S, rel_tol, max_iter);
        bi_update<<<nb, kBlock, 0, ss>>>(m, phi, r, rhat, p, sv, t, part, part2, S);
        bi_scalars<<<1, kBlock, 0, ss>>>(3, part, part2, nb, S, rel_tol, max_iter);
    });
    if (rc) return rc;
    if (iterations) *iterations = (int64_t)host[bITERS];
    if (rel_residual) *rel_residual = host[bBB] > 0.0 ? std::sqrt(host[bRR] / host[bBB]) : 0.0;
    return PPT_OK;
}

extern "C" int ppt_poisson_solve_coef(const ppt_mesh_desc* mesh, const double* coef, const double* rhs, double* phi,
                                      void* scratch, double rel_tol, int64_t max_iter, int64_t* iterations,
                                      double* rel_residual, void* stream) {
    return solve_coef(mesh, coef, rhs, phi, scratch, rel_tol, max_iter, kSpinLimit, iterations, rel_residual, stream);
}

// The two solves (coef NULL: the first) with waits of at most `polls` polls, how a
// test makes one run out, or (0) with the cooperative launch refused.  Not part of
// the library's interface.
extern "C" int ppt_poisson_solve_polls(const ppt_mesh_desc* mesh, const double* coef, const double* rhs, double* phi,
                                       void* scratch, double rel_tol, int64_t max_iter, int polls, void* stream) {
    if (coef) return solve_coef(mesh, coef, rhs, phi, scratch, rel_tol, max_iter, polls, nullptr, nullptr, stream);
    return solve_laplacian(mesh, rhs, phi, scratch, rel_tol, max_iter, polls, nullptr, nullptr, stream);
}
