// Plain form: the reference's pushers in float64, fused with the trilinear
// gathers, many steps per launch.
//
// One thread owns one particle for the whole launch.  Its position and
// velocity live in registers across all steps of the call; per step it
// locates its cell, gathers the 8 corner records (one 256-bit load per field
// per corner), interpolates E and B, applies the algorithm's update and
// writes a snapshot row only on record steps.  The reference instead makes 6
// (Boris/Vay) or 24 (RK4) separate interpolation passes per step over
// particle arrays in DRAM, each with its own binary search
// (src/PyPATools/pusher.py:966-980, :699-801, field.py:491-504).
//
// Arithmetic follows the reference's kernels term by term so the results
// agree to rounding: Boris pusher.py:124-165, Vay 'vay_rel' :216-279,
// relativistic gamma :74-96, RK4 :803-892 with derivatives :168-172 and
// :282-298, leapfrog :730-739, Yoshida :184-209 / :332-362 (fields frozen at
// the step start), |v| clamps :275-277 / :886-890.  boris_rel and vay are
// additions (u = gamma v state, see the oracle for their equations).
#pragma once

#include <cmath>

#include "track_params.cuh"

namespace ppt {


__host__ __device__ constexpr bool alg_staggered(int a) {
    return a == PPT_ALG_BORIS || a == PPT_ALG_BORIS_REL || a == PPT_ALG_VAY;
}
__host__ __device__ constexpr bool alg_u_state(int a) { return a == PPT_ALG_BORIS_REL || a == PPT_ALG_VAY; }

// Yoshida (1990) 4th-order coefficients, the float64 values of the
// reference's expressions (pusher.py:176-181), written to round-trip exactly.
constexpr double kYoC1 = 1.3512071919596578;     // 1 / (2 - 2^(1/3))
constexpr double kYoC2 = -1.7024143839193153;    // -2^(1/3) / (2 - 2^(1/3))
constexpr double kYoD1 = 2.7024143839193155;     // 2 C1
constexpr double kYoD2 = -3.0536215758789735;    // -(2^(1/3) + 1) / (2 - 2^(1/3))

// ---------------------------------------------------------------------------
// per-algorithm updates (float64)
// ---------------------------------------------------------------------------
// The relativistic updates below are bound by instruction issue and by the
// latency of their one serial chain (18-23 % occupancy at their register
// counts), and most of their instructions were float64 divisions (about ten
// instructions each, and a branch): by c, by c^2, by gamma, by gamma_new.
// They are written in 1/gamma instead -- sqrt(1 - beta^2), or one rsqrt --
// with 1/c and 1/c^2 as constants, |v| compared by its square, and each sum
// of products as explicit FMAs, so a layout that leaves zero components out
// (EM, BM masks) computes the bits of the full form: fma(a, 0, s) is s, and a
// chain's first product is rounded on its own (__dmul_rn) where the full
// form adds it to an exact zero.
// Measured (kernel time): 1e6 electrons x 200 rk4_rel steps 18.4 -> 15.3 ms,
// 4e5 x 500 vay_rel steps 4.88 -> 3.79 ms; the error against float64 torch is
// unchanged (2.5e-14 and 5.4e-13).
constexpr double kInvC = 1.0 / kClight;
constexpr double kInvC2 = 1.0 / (kClight * kClight);

__device__ __forceinline__ double dot_fma(V3 a, V3 b) { return fma(a.z, b.z, fma(a.y, b.y, __dmul_rn(a.x, b.x))); }

// a.b without the components outside M (exact zeros of either vector)
template <int M>
__device__ __forceinline__ double dot_m(V3 a, V3 b) {
    if constexpr (M == 0) return 0.0;
    else if constexpr (M == 4) return __dmul_rn(a.z, b.z);
    else if constexpr (M == 2) return __dmul_rn(a.y, b.y);
    else if constexpr (M == 6) return fma(a.z, b.z, __dmul_rn(a.y, b.y));
    else {
        double s = __dmul_rn(a.x, b.x);
        if constexpr (bit(M, 1)) s = fma(a.y, b.y, s);
        if constexpr (bit(M, 2)) s = fma(a.z, b.z, s);
        return s;
    }
}

// s + p x q, component by component, without q's components outside QM
template <int QM>
__device__ __forceinline__ V3 add_cross(V3 s, V3 p, V3 q) {
    if constexpr (bit(QM, 1)) {
        s.x = fma(-p.z, q.y, s.x);
        s.z = fma(p.x, q.y, s.z);
    }
    if constexpr (bit(QM, 2)) {
        s.x = fma(p.y, q.z, s.x);
        s.y = fma(-p.x, q.z, s.y);
    }
    if constexpr (bit(QM, 0)) {
        s.y = fma(p.z, q.x, s.y);
        s.z = fma(-p.y, q.x, s.z);
    }
    return s;
}

__device__ __forceinline__ V3 axpy(double a, V3 x, V3 y) { return v3(fma(a, x.x, y.x), fma(a, x.y, y.y), fma(a, x.z, y.z)); }

// a x + y on the components x can have (M)
template <int M>
__device__ __forceinline__ V3 axpy_m(double a, V3 x, V3 y) {
    if constexpr (bit(M, 0)) y.x = fma(a, x.x, y.x);
    if constexpr (bit(M, 1)) y.y = fma(a, x.y, y.y);
    if constexpr (bit(M, 2)) y.z = fma(a, x.z, y.z);
    return y;
}

// a x on the components x can have (M), zeros elsewhere
template <int M>
__device__ __forceinline__ V3 scale_m(double a, V3 x) {
    return v3(bit(M, 0) ? a * x.x : 0.0, bit(M, 1) ? a * x.y : 0.0, bit(M, 2) ? a * x.z : 0.0);
}

// u + (w + p x q) with q's components in QM (and w's no others): the small terms
// first, so that u is rounded once.  A step adds a hundredth of u or less, and what
// is rounded off at the size of u, term by term, stays in the track.
template <int QM>
__device__ __forceinline__ V3 add_small(V3 u, V3 w, V3 p, V3 q) {
    const V3 d = add_cross<QM>(w, p, q);
    constexpr int M = QM | cross_bits(QM);
    if constexpr (bit(M, 0)) u.x += d.x;
    if constexpr (bit(M, 1)) u.y += d.y;
    if constexpr (bit(M, 2)) u.z += d.z;
    return u;
}

// beta^2, at most 0.9999 (pusher.py:74-96)
__device__ __forceinline__ double clamped_beta2(V3 v) {
    const double bsq = dot_fma(v, v) * kInvC2;
    return bsq >= 0.9999 ? 0.9999 : bsq;
}

__device__ __forceinline__ V3 clamp_speed(V3 v) {
    constexpr double top = 0.9999 * kClight;
    const double v2 = dot_fma(v, v);
    // (also where v2 is NaN: every component is then, whatever the record layout leaves out)
    if (!(v2 < top * top)) v = v * (top * rsqrt(v2));
    return v;
}


// (p x q)_I in the reference's form p_J q_K - p_K q_J, without q's components
// outside the mask QM (an exact zero there).  A lone product is rounded on
// its own (__dmul_rn), as the full form rounds it before the caller adds it
// to a vector: left to the compiler, v + p_J q_K would fuse into one FMA and
// round once, which the full form never does.
template <int QM, int I>
__device__ __forceinline__ double cross_md(const double p[3], const double q[3]) {
    constexpr int J = (I + 1) % 3, K = (I + 2) % 3;
    if constexpr (bit(QM, K) && bit(QM, J)) return p[J] * q[K] - p[K] * q[J];
    else if constexpr (bit(QM, K)) return __dmul_rn(p[J], q[K]);
    else if constexpr (bit(QM, J)) return -__dmul_rn(p[K], q[J]);
    else return 0.0;
}

// boris_v for fields whose components outside EM (E) and BM (B) are zero by
// construction (a single map of a pruned record layout, no constant parts):
// the same operations on the components that can be non-zero, none on the
// others (pusher.py:124-165).
template <int EM, int BM>
__device__ __forceinline__ V3 boris_v_m(V3 v, V3 E, V3 B, double dt, double qm) {
    constexpr int CM = cross_bits(BM);
    const double h = 0.5 * qm;
    const double vv[3] = {v.x, v.y, v.z}, e[3] = {E.x, E.y, E.z}, b[3] = {B.x, B.y, B.z};
    double kick[3], vm[3], t[3], s[3], vp[3], out[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        kick[i] = bit(EM, i) ? h * e[i] * dt : 0.0;
        vm[i] = bit(EM, i) ? vv[i] + kick[i] : vv[i];
        t[i] = bit(BM, i) ? h * b[i] * dt : 0.0;
    }
    // t.t: a lone square rounded on its own, as the full form's sum rounds it
    // (left to the compiler, 1 + t_z t_z would fuse into one FMA)
    double tt;
    if constexpr (BM == 0) tt = 0.0;
    else if constexpr (BM == 4) tt = __dmul_rn(t[2], t[2]);
    else if constexpr (BM == 1) tt = __dmul_rn(t[0], t[0]);
    else if constexpr (BM == 2) tt = __dmul_rn(t[1], t[1]);
    else tt = t[0] * t[0] + t[1] * t[1] + t[2] * t[2];
    const double f = 2.0 / (1.0 + tt);
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] = bit(BM, i) ? t[i] * f : 0.0;
    vp[0] = bit(CM, 0) ? vm[0] + cross_md<BM, 0>(vm, t) : vm[0];
    vp[1] = bit(CM, 1) ? vm[1] + cross_md<BM, 1>(vm, t) : vm[1];
    vp[2] = bit(CM, 2) ? vm[2] + cross_md<BM, 2>(vm, t) : vm[2];
    const double c2[3] = {cross_md<BM, 0>(vp, s), cross_md<BM, 1>(vp, s), cross_md<BM, 2>(vp, s)};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double vplus = bit(CM, i) ? vm[i] + c2[i] : vm[i];
        out[i] = bit(EM, i) ? vplus + kick[i] : vplus;
    }
    return v3(out[0], out[1], out[2]);
}

// The reference's Boris (pusher.py:124-165): kick = (q/m) E dt / 2,
// v- = v + kick, t = (q/m) B dt / 2, s = 2 t / (1 + t.t), v' = v- + v- x t,
// v+ = v- + v' x s, v_new = v+ + kick -- the masked form with every
// component present, so a map of a pruned record layout computes the same
// bits as one that stores its zero components.
__device__ __forceinline__ V3 boris_v(V3 v, V3 E, V3 B, double dt, double qm) {
    return boris_v_m<7, 7>(v, E, B, dt, qm);
}

// The reference's 'vay_rel' (pusher.py:216-279) in u = gamma v:
// gn^2 = (sigma + sqrt(sigma^2 + 4 (tau^2 + u*^2))) / 2, t = tau / gn,
// s = 2 t / (1 + t.t), v = (u' + (u' + u' x t) x s) / gn.
template <int EM, int BM>
__device__ __forceinline__ V3 vay_rel_v(V3 v, V3 E, V3 B, double dt, double qm) {
    const double qdt = qm * dt, h = 0.5 * qdt;
    const V3 tau = h * B;
    // gamma v + (q/m) E dt in one rounding: with u = gamma v rounded by itself, a kick
    // far below u meets the same rounding at every step of a straight track
    const V3 up = axpy(rsqrt(1.0 - clamped_beta2(v)), v, scale_m<EM>(qdt, E));
    const double tau2 = dot_m<BM>(tau, tau);
    const double q = dot_fma(up, tau) * kInvC;
    double gis = fma(-dot_fma(up, up), kInvC2, 1.0);
    if (gis < 1e-10) gis = 1e-10;
    const double sigma = gis - tau2;
    const double ig = rsqrt(0.5 * (sigma + sqrt(fma(sigma, sigma, 4.0 * fma(q, q, tau2)))));
    const V3 t = ig * tau;
    const V3 s = (2.0 / fma(tau2, ig * ig, 1.0)) * t;
    const V3 us = add_cross<BM>(up, up, t);
    return clamp_speed(ig * add_cross<BM>(up, us, s));
}

// (every product is formed: a velocity component that is not finite reaches
// the others through the zero components of B, as in the reference)
__device__ __forceinline__ V3 lorentz(V3 v, V3 E, V3 B, double qm) { return qm * add_cross<7>(E, v, B); }

// dv/dt = ((q/m) F - v (v . (q/m) F) / c^2) / gamma, F = E + v x B
// (pusher.py:282-298), with 1/gamma = sqrt(1 - beta^2).
template <int EM, int BM>
__device__ __forceinline__ V3 rk4_rel_deriv(V3 v, V3 E, V3 B, double qm) {
    constexpr int FM = EM | cross_bits(BM);
    const double k = qm * sqrt(1.0 - clamped_beta2(v));
    const V3 F = add_cross<BM>(E, v, B);
    const double s = dot_m<FM>(v, F) * kInvC2;
    return k * axpy(-s, v, F);
}

// 1 / gamma of u = gamma v
__device__ __forceinline__ double inv_gamma_u(V3 u) { return rsqrt(fma(dot_fma(u, u), kInvC2, 1.0)); }

template <int EM, int BM>
__device__ __forceinline__ V3 boris_rel_u(V3 u, V3 E, V3 B, double dt, double qm) {
    const double h = 0.5 * qm * dt;
    const V3 um = axpy_m<EM>(h, E, u);
    const V3 t = (h * inv_gamma_u(um)) * B;
    const V3 s = (2.0 / (1.0 + dot_m<BM>(t, t))) * t;
    const V3 up = add_cross<BM>(um, um, t);
    return axpy_m<EM>(h, E, add_small<BM>(um, v3(0.0, 0.0, 0.0), up, s));
}

// Vay (2008); v_old = u / gamma(u).
template <int EM, int BM>
__device__ __forceinline__ V3 vay_u(V3 u, V3 v_old, V3 E, V3 B, double dt, double qm) {
    const double h = 0.5 * qm * dt;
    // u' = u + (q/m) dt (E + v x B / 2), the increment added to u once
    const V3 tau = h * B;
    const V3 up = axpy_m<EM | cross_bits(BM)>(h, add_cross<BM>(scale_m<EM>(2.0, E), v_old, B), u);
    const double tau2 = dot_m<BM>(tau, tau);
    const double us = dot_m<BM>(up, tau) * kInvC;
    const double sigma = fma(dot_fma(up, up), kInvC2, 1.0) - tau2;
    const double ig = rsqrt(0.5 * (sigma + sqrt(fma(sigma, sigma, 4.0 * fma(us, us, tau2)))));
    const V3 t = ig * tau;
    const double s = 1.0 / fma(tau2, ig * ig, 1.0);
    return s * add_small<BM>(up, scale_m<BM>(dot_m<BM>(up, t), t), up, t);
}

template <int ALG>
__device__ __forceinline__ V3 w_to_v(V3 w) {
    if constexpr (alg_u_state(ALG)) return inv_gamma_u(w) * w;
    else return w;
}

// Components a launch's E and B can have: those of its record layout, all for
// the run-time dispatch (L = 0).
__host__ __device__ constexpr int launch_e_bits(int L) { return L == 0 ? 7 : e_bits(L); }
__host__ __device__ constexpr int launch_b_bits(int L) { return L == 0 ? 7 : b_bits(L); }

template <int ALG, int L>
__device__ __forceinline__ V3 half_kick(V3 w, V3 E, V3 B, double dt, double qm) {
    constexpr int EM = launch_e_bits(L), BM = launch_b_bits(L);
    if constexpr (ALG == PPT_ALG_BORIS) return boris_v(w, E, B, dt, qm);
    else if constexpr (ALG == PPT_ALG_BORIS_REL) return boris_rel_u<EM, BM>(w, E, B, dt, qm);
    else return vay_u<EM, BM>(w, w_to_v<ALG>(w), E, B, dt, qm);
}

// The 8 corner records of one cell of a single-layout map, for the kernels
// that keep them in registers from one field evaluation to the next
// (keeps_corners below).  Corner q = di*4 + dj*2 + dk; the pad of a
// four-element record is not kept.
__host__ __device__ constexpr int layout_slots(int L) { return layout_width(L) == 4 ? 3 : layout_width(L); }

template <int L>
struct Corners {
    int64_t base = -1;                 // node index of corner (0, 0, 0), -1: none
    double v[8][layout_slots(L)];
};
template <>
struct Corners<0> {};

template <int L>
__device__ __forceinline__ void load_corners(const MapDev& m, int64_t base, Corners<L>& K) {
    constexpr int W = layout_width(L);
    static_assert(W <= 4, "the six-component record is gathered field by field");
    const double* p = static_cast<const double*>(m.data) + base * W;
    const int64_t sx = m.sx * W, sy = m.sy * W;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double* c = p + ((q >> 2) & 1) * sx + ((q >> 1) & 1) * sy + (q & 1) * W;
        if constexpr (W == 4) {
            double pad;
            ldg_f64x4(c, K.v[q][0], K.v[q][1], K.v[q][2], pad);
        } else if constexpr (W == 2) {
            ldg_f64x2(c, K.v[q][0], K.v[q][1]);
        } else {
            K.v[q][0] = __ldg(c);
        }
    }
    K.base = base;
}

// E and B from the kept corners: tri() per stored component.
template <int L>
__device__ __forceinline__ void interp_corners(const Corners<L>& K, const Cell& c, V3& E, V3& B) {
    constexpr int S = layout_slots(L);
    double o[S];
#pragma unroll
    for (int k = 0; k < S; ++k)
        o[k] = tri(K.v[0][k], K.v[4][k], K.v[2][k], K.v[6][k], K.v[1][k], K.v[5][k], K.v[3][k], K.v[7][k], c.tx, c.ty,
                   c.tz);
    if constexpr (L == kLayE) E = v3(o[0], o[1], o[2]);
    else if constexpr (L == kLayB) B = v3(o[0], o[1], o[2]);
    else if constexpr (L == kLayExEyBz) {
        E = v3(o[0], o[1], 0.0);
        B = v3(0.0, 0.0, o[2]);
    } else if constexpr (L == kLayEzBz) {
        E = v3(0.0, 0.0, o[0]);
        B = v3(0.0, 0.0, o[1]);
    } else {
        B = v3(0.0, 0.0, o[0]);
    }
}

// Which kernels keep the corner records between field evaluations.  RK4's
// four evaluations of a step lie within one step's advance of each other (the
// two middle ones almost coincide, and the last is next to the next step's
// first), so most of its lanes find their cell unchanged and load nothing:
// the L1 wavefronts of incoherent gathers are what bounds it.  The same holds
// for Vay's one evaluation a step while a step is short against a cell.  The
// Boris kernels are bound by issue, where a load that most lanes skip still
// takes its slots, and run 6 blocks per SM on 80 registers: not there, nor for
// the six-component record (96 registers).  Measured, kernel time: 1e6
// electrons x 200 rk4_rel steps 15.3 -> 6.99 ms (L1 was at 80 %), 4e5 x 500
// vay_rel steps 3.85 -> 2.87, vay 4.72 -> 2.73; protons of the ring, which change
// their cell every step, 5e5 x 100 rk4_rel steps 1.46 -> 1.34, vay_rel 0.63 -> 0.60.
__host__ __device__ constexpr bool keeps_corners(int alg, int L) {
    return L != 0 && L != kLayFull &&
           (alg == PPT_ALG_RK4 || alg == PPT_ALG_RK4_REL || alg == PPT_ALG_VAY || alg == PPT_ALG_VAY_REL);
}

struct Ctx {
    const FieldsDev* F;
    double dt, qm, omega, phase, t0;
    unsigned hits;
    int const_nz;
    double c0, s0;            // cos, sin of omega t0 + phase
    const double2* tab;       // (cos, sin) of g omega dt for the launch's steps, or NULL
    int64_t tab0;             // the launch's first step
};

// Per-step RF table length limit (shared memory, 16 B per step): the sorted
// launches of a bunch crossing its map are a few hundred steps; longer
// launches evaluate the same expression directly.
constexpr int kRfTable64 = 512;

// Fill the block's table of (cos, sin) of g omega dt for steps step0 ..
// step0 + n - 1 (all threads of the block call it; n <= kRfTable64).
__device__ __forceinline__ void build_rf_table64(double2* tab, int64_t step0, int n, double wdt) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double sg, cg;
        sincos((double)(step0 + i) * wdt, &sg, &cg);
        tab[i] = make_double2(cg, sg);
    }
    __syncthreads();
}

// E and B of a single uniform-grid map of record layout L with no constant
// parts (E, B zero outside it); returns 1 when r is inside.  The cell search
// is locate_axis's uniform branch, the interpolation tri() per stored
// component, so the values are the run-time dispatch's (eval_fields_f64).
// (KEEP: K holds the cell of the last evaluation, and a point in the same
// cell loads nothing.)
template <int L, bool KEEP>
__device__ __forceinline__ int eval_single_f64(const MapDev& m, V3 r, V3& E, V3& B, Corners<KEEP ? L : 0>& K) {
    E = v3(0.0, 0.0, 0.0);
    B = v3(0.0, 0.0, 0.0);
    if (!(axis_contains(m.ax[0], r.x) & axis_contains(m.ax[1], r.y) & axis_contains(m.ax[2], r.z))) return 0;
    Cell c;
    int ijk[3];
    double tt[3];
    const double x[3] = {r.x, r.y, r.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u = __dmul_rn(x[a] - m.ax[a].lo, m.ax[a].inv_d);
        ijk[a] = __double2int_rd(u);             // floor: u is in [0, n - 1] here
        tt[a] = u - (double)ijk[a];
    }
    // cells 1 .. n-3 on every axis need none of the clamps below (the cell is
    // in range and u - floor(u) is in [0, 1)); the others take them
    if (!(((unsigned)(ijk[0] - 1) < (unsigned)(m.ax[0].n - 3)) & ((unsigned)(ijk[1] - 1) < (unsigned)(m.ax[1].n - 3)) &
          ((unsigned)(ijk[2] - 1) < (unsigned)(m.ax[2].n - 3)))) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const AxisDev& ax = m.ax[a];
            const double u = __dmul_rn(x[a] - ax.lo, ax.inv_d);
            int cc = ijk[a];
            cc = cc < 0 ? 0 : (cc > ax.n - 2 ? ax.n - 2 : cc);
            const double t = u - (double)cc;
            tt[a] = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
            ijk[a] = cc;
        }
    }
    c.tx = tt[0];
    c.ty = tt[1];
    c.tz = tt[2];
    c.base = (int64_t)ijk[0] * m.sx + (int64_t)ijk[1] * m.sy + ijk[2];
    if constexpr (L == kLayFull) {
        E = gather_f64s<8>(m, c, 0);
        B = gather_f64s<8>(m, c, 4);
    } else if constexpr (KEEP) {
        if (c.base != K.base) load_corners<L>(m, c.base, K);
        interp_corners<L>(K, c, E, B);
    } else {
        Corners<L> now;
        load_corners<L>(m, c.base, now);
        interp_corners<L>(now, c, E, B);
    }
    return 1;
}

// Fields at r and field time t0 + g dt + toff; the time and the RF cosine are
// only formed when E is non-zero.  Returns the number of maps containing r.
// L = 0: any fields (maps summed at run time, constant parts); otherwise a
// single map of record layout L (eval_single_f64).
// RF factor cos(omega (t0 + g dt + toff) + phi): at the step's own time
// (toff = 0) as cos(a + b) = cos a cos b - sin a sin b with a = omega t0 + phi
// per particle and b = g omega dt per step, (cos b, sin b) from the launch's
// table or, beyond it, the same float64 expression, so a track's bits do not
// depend on how it is split into launches; at RK4's stage times directly.
template <bool RF, int L, bool KEEP = false>
__device__ __forceinline__ int fields_at(Ctx& c, V3 r, int64_t g, double toff, V3& E, V3& B,
                                         Corners<KEEP ? L : 0>& K) {
    int h;
    if constexpr (L == 0) h = eval_fields_f64(*c.F, r, E, B);
    else h = eval_single_f64<L, KEEP>(c.F->maps[0], r, E, B, K);
    c.hits += h;
    if (RF) {
        constexpr int EM = L == 0 ? 7 : e_bits(L);
        if ((bit(EM, 0) && E.x != 0.0) || (bit(EM, 1) && E.y != 0.0) || (bit(EM, 2) && E.z != 0.0)) {
            double cf;
            if (toff == 0.0) {
                double cg, sg;
                if (c.tab != nullptr) {
                    const double2 t = c.tab[g - c.tab0];
                    cg = t.x;
                    sg = t.y;
                } else {
                    sincos((double)g * (c.omega * c.dt), &sg, &cg);
                }
                cf = fma(c.c0, cg, -(c.s0 * sg));
            } else {
                const double t = c.t0 + (double)g * c.dt + toff;
                cf = cos(c.omega * t + c.phase);
            }
            if constexpr (bit(EM, 0)) E.x = E.x * cf;
            if constexpr (bit(EM, 1)) E.y = E.y * cf;
            if constexpr (bit(EM, 2)) E.z = E.z * cf;
        }
    }
    return h;
}

template <bool RF, int L>
__device__ __forceinline__ int fields_at(Ctx& c, V3 r, int64_t g, double toff, V3& E, V3& B) {
    Corners<0> none;
    return fields_at<RF, L, false>(c, r, g, toff, E, B, none);
}

// Position advance of one step, r + v dt (pusher.py:395-404).
__device__ __forceinline__ V3 drift(V3 r, V3 v, double dt) {
    return v3(fma(v.x, dt, r.x), fma(v.y, dt, r.y), fma(v.z, dt, r.z));
}

// m field-free steps of one coordinate, x <- fma(v, dt, x) at each, with the
// bits of the step-by-step loop.  The float64 numbers whose magnitude lies
// in one binade [2^E, 2^(E+1)) are the multiples of g = 2^(E-52) there, and x
// is one of them; so when the exact sum x + v dt lies in x's binade it rounds
// to x + D, D being v dt rounded to a multiple of g -- the same D at every
// such step, unless v dt lies exactly halfway between two multiples (then
// round-half-even looks at x's last bit).  Each trip of the loop therefore
// takes the steps whose sums certainly stay inside x's binade as k D in one
// exact fused multiply-add, then one step as it comes (the step out of the
// binade, a halfway case, or a step within four steps of zero).  A
// coordinate crossing zero passes the binades between |v dt| and |x| one
// trip each.
__device__ __forceinline__ double drift_coord(double x, double v, double dt, int m) {
    // a zero advance: the first step settles the sign of a zero x, the others keep x
    if (v == 0.0 || dt == 0.0) return m > 0 ? fma(v, dt, x) : x;
    const double p = v * dt;
    const double ap = fabs(p) * (1.0 + 0x1p-50);   // above |v dt| exactly
    while (m > 0) {
        const double ax = fabs(x);
        // (false for NaN and infinities too)
        if (ax >= 4.0 * ap && ax >= 0x1p-64 && ax < 0x1p1000) {
            const long long eb = __double_as_longlong(ax) >> 52;    // biased exponent of |x|
            const double lo = __longlong_as_double(eb << 52);        // 2^E
            const double D = fma(v, dt, x) - x;   // exact: the sum lies within [x/2, 2x]
            // distance of the sums from the binade's edge ahead, from below
            const double room = ((p > 0.0) == (x > 0.0) ? 2.0 * lo - ax : ax - lo) - ap;
            // not halfway: |v dt - D| != g / 2 = 2^(E-53)
            if (room > 0.0 && fabs(fma(v, dt, -D)) != __longlong_as_double((eb - 53) << 52)) {
                // steps n = 0 .. k-1 with n |D| < room; the quotient's error
                // (a few float32 ulps) is far inside the 1e-4 margin
                int k = m;
                if (D != 0.0) {
                    const float kq = __fdividef((float)room, (float)fabs(D)) * 0.9999f;
                    if (!(kq >= (float)m)) k = kq >= 1.0f ? (int)kq : 1;
                }
                x = fma((double)k, D, x);
                m -= k;
                if (m == 0) break;
            }
        }
        x = fma(v, dt, x);
        --m;
    }
    return x;
}

// A short run is quicker step by step: three independent FMAs a step, against
// some hundred dependent instructions per coordinate (one proton, 1000 steps of
// which 640 are field-free, kernel time with a record every 1 / 7 / 20 / 50
// steps: 790 / 243 / 183 / 165 us closed form, 392 / 192 / 170 / 164 with runs of
// up to 32 steps taken so).
constexpr int kShortRun = 32;

__device__ __forceinline__ V3 drift_run(V3 r, V3 v, double dt, int m) {
    if (m <= kShortRun) {
        for (; m > 0; --m) r = drift(r, v, dt);
        return r;
    }
    return v3(drift_coord(r.x, v.x, dt, m), drift_coord(r.y, v.y, dt, m), drift_coord(r.z, v.z, dt, m));
}

__host__ __device__ constexpr bool alg_skips_free(int a) {
    return a == PPT_ALG_LEAPFROG || a == PPT_ALG_BORIS || a == PPT_ALG_BORIS_REL;
}

// Steps a particle moving at v certainly stays outside every map, so that
// they are field-free drift steps (only for fields without constant parts):
// outside the union box of the maps on some axis, it must travel `dist` at
// `rate` per step to come back on that axis.  After j steps the position
// carries at most j * 2^-53 * X of rounding (X bounds |x| on the way), which
// the margin covers.
__device__ __forceinline__ int quiet_steps_f64(const FieldsDev& F, V3 r, V3 v, double dt) {
    if (F.n_maps == 0) return 0;
    const double x[3] = {r.x, r.y, r.z}, u[3] = {v.x * dt, v.y * dt, v.z * dt};
    double best = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double dist, rate, bound;
        if (x[a] < F.box_lo[a]) {
            dist = F.box_lo[a] - x[a];
            rate = u[a];
            bound = F.box_lo[a];
        } else if (x[a] > F.box_hi[a]) {
            dist = x[a] - F.box_hi[a];
            rate = -u[a];
            bound = F.box_hi[a];
        } else {
            continue;
        }
        const double X = fmax(fabs(x[a]), fabs(bound));
        const double k = rate > 0.0 ? dist / (rate + 2.3e-16 * X) : 2e9;
        best = fmax(best, k);
    }
    best = best * (1.0 - 1e-9) - 2.0;
    return best <= 0.0 ? 0 : (best >= 1e9 ? 1000000000 : (int)best);
}

// One step; returns true for a field-free step of the Boris family (its
// velocity update skipped, see below).
// (vel: the velocity of the state w, kept between the steps of the u-state
// algorithms, whose drift forms it anyway.)
template <int ALG, bool RF, int L>
__device__ __forceinline__ bool step(Ctx& c, V3& r, V3& w, V3& vel, int64_t g,
                                     Corners<keeps_corners(ALG, L) ? L : 0>& K) {
    constexpr bool KEEP = keeps_corners(ALG, L);
    constexpr int EM = launch_e_bits(L), BM = launch_b_bits(L);
    const double dt = c.dt, qm = c.qm;
    if constexpr (ALG == PPT_ALG_RK4 || ALG == PPT_ALG_RK4_REL) {
        constexpr bool REL = ALG == PPT_ALG_RK4_REL;
        V3 E, B;
        const double h = 0.5 * dt;
        fields_at<RF, L, KEEP>(c, r, g, 0.0, E, B, K);
        V3 k1v = REL ? rk4_rel_deriv<EM, BM>(w, E, B, qm) : lorentz(w, E, B, qm);
        V3 k1r = w;
        V3 r2 = axpy(h, k1r, r), v2 = axpy(h, k1v, w);
        fields_at<RF, L, KEEP>(c, r2, g, h, E, B, K);
        V3 k2v = REL ? rk4_rel_deriv<EM, BM>(v2, E, B, qm) : lorentz(v2, E, B, qm);
        V3 r3 = axpy(h, v2, r), v3_ = axpy(h, k2v, w);
        fields_at<RF, L, KEEP>(c, r3, g, h, E, B, K);
        V3 k3v = REL ? rk4_rel_deriv<EM, BM>(v3_, E, B, qm) : lorentz(v3_, E, B, qm);
        V3 r4 = axpy(dt, v3_, r), v4 = axpy(dt, k3v, w);
        fields_at<RF, L, KEEP>(c, r4, g, dt, E, B, K);
        V3 k4v = REL ? rk4_rel_deriv<EM, BM>(v4, E, B, qm) : lorentz(v4, E, B, qm);
        const double s6 = dt / 6.0;
        r = axpy(s6, axpy(2.0, v3_, axpy(2.0, v2, k1r)) + v4, r);
        w = axpy(s6, axpy(2.0, k3v, axpy(2.0, k2v, k1v)) + k4v, w);
        if (REL) w = clamp_speed(w);
    } else if constexpr (ALG == PPT_ALG_YOSHIDA || ALG == PPT_ALG_YOSHIDA_REL) {
        constexpr bool REL = ALG == PPT_ALG_YOSHIDA_REL;
        V3 E, B;
        fields_at<RF, L, KEEP>(c, r, g, 0.0, E, B, K);
        const double cs[3] = {kYoC1, kYoC2, kYoC1};
        const double ds[3] = {kYoD1, kYoD2, kYoD1};
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            V3 a = REL ? rk4_rel_deriv<EM, BM>(w, E, B, qm) : lorentz(w, E, B, qm);
            w = w + (cs[s] * dt) * a;
            r = r + (ds[s] * dt) * w;
        }
        if (REL) w = clamp_speed(w);
    } else {
        V3 E, B;
        // With no map containing r and no constant field, E = B = 0 exactly and
        // the leapfrog, Boris and relativistic Boris updates return w unchanged
        // (every term they add is a signed zero), so they are skipped.
        const bool any = fields_at<RF, L, KEEP>(c, r, g, 0.0, E, B, K) != 0 || c.const_nz;
        if constexpr (ALG == PPT_ALG_LEAPFROG) {
            if (any) w = axpy(dt, lorentz(w, E, B, qm), w);
            r = drift(r, w, dt);
        } else if constexpr (ALG == PPT_ALG_BORIS) {
            if (any) {
                if constexpr (L == 0) w = boris_v(w, E, B, dt, qm);
                else w = boris_v_m<e_bits(L), b_bits(L)>(w, E, B, dt, qm);
            }
            r = drift(r, w, dt);
        } else if constexpr (ALG == PPT_ALG_VAY_REL) {
            w = vay_rel_v<EM, BM>(w, E, B, dt, qm);
            r = drift(r, w, dt);
        } else if constexpr (ALG == PPT_ALG_BORIS_REL) {
            // (unchanged u, unchanged velocity)
            if (any) {
                w = boris_rel_u<EM, BM>(w, E, B, dt, qm);
                vel = w_to_v<ALG>(w);
            }
            r = drift(r, vel, dt);
        } else {  // PPT_ALG_VAY
            w = vay_u<EM, BM>(w, vel, E, B, dt, qm);
            vel = w_to_v<ALG>(w);
            r = drift(r, vel, dt);
        }
        return alg_skips_free(ALG) && !any;
    }
    return false;
}

// The velocity of state w, for the snapshot rows and the field-free runs.
template <int ALG>
__device__ __forceinline__ V3 state_velocity(V3 w, V3 vel) {
    if constexpr (alg_u_state(ALG)) return vel;
    else return w;
}

__device__ __forceinline__ double* row_at(double* hist, int64_t rec, int64_t n, int64_t row) {
    return hist + (rec * n + row) * 3;
}

__device__ __forceinline__ void write_row(double* p, V3 a) {
    p[0] = a.x;
    p[1] = a.y;
    p[2] = a.z;
}

__device__ __forceinline__ Ctx make_ctx(const TrackDev& P) {
    return Ctx{&P.F, P.dt, P.qm, P.omega, 0.0, P.t0, 0u, P.F.e_const_nz | P.F.b_const_nz, 1.0, 0.0, nullptr, 0};
}

// All steps of one call for particle slot s (s < P.n); returns the steps done.
// COLL: each step's segment is tested against the electrode surface after the
// step's snapshot, and a particle that hits stops there (pusher.py:966-990).
// Measured (kernel time, 1e6 protons x 1000 steps through a pipe and an aperture
// plate, most of them stopped within 300): 15.1 ms with the test of every
// triangle listed by a step's cells, 10.6 with the plane test in front of it and
// clear boxes (surface.cuh), 7.2 on the refined segment grid.
template <int ALG, bool RF, bool COLL, int L>
__device__ __forceinline__ unsigned track_f64_particle(const TrackDev& P, int64_t s, Ctx& c) {
    {
        const int64_t n = P.n;
        double* st = P.f64;
        const int64_t row = P.order ? P.order[s] : s;
        if constexpr (COLL) {
            if (!P.active[row]) return 0;   // stopped in an earlier call: nothing moves or records
        }
        V3 r = v3(st[s], st[n + s], st[2 * n + s]);
        V3 w = v3(st[3 * n + s], st[4 * n + s], st[5 * n + s]);
        if constexpr (ALG == PPT_ALG_RK4 || ALG == PPT_ALG_RK4_REL) {
            // the reference's array dt: every stage of this particle's step uses its own
            // dt (pusher.py:815-816), and so does its field time t0 + g dt (the
            // launch's RF table holds the launch's dt: not used then)
            if (P.dt_rows) {
                c.dt = P.dt_rows[row];
                c.tab = nullptr;
            }
        }
        if (RF) {
            c.phase = P.rf_phase[s];
            double sa, ca;
            sincos(fma(c.omega, c.t0, c.phase), &sa, &ca);
            c.c0 = ca;
            c.s0 = sa;
        }
        bool stopped = false;

        if (P.flags & PPT_TRACK_INIT) {
            if constexpr (alg_staggered(ALG)) {
                V3 E, B;
                fields_at<RF, L>(c, r, P.step0, 0.0, E, B);
                w = half_kick<ALG, L>(w, E, B, -0.5 * P.dt, P.qm);
            }
            if (P.r_hist) {
                write_row(row_at(P.r_hist, 0, n, row), r);
                write_row(row_at(P.v_hist, 0, n, row), w_to_v<ALG>(w));
            }
        }
        V3 vel = w_to_v<ALG>(w);
        Corners<keeps_corners(ALG, L) ? L : 0> K;
        // steps until the next record: record after global step g when (g+1) % rec == 0;
        // the records are numbered by counting on from the launch's first (with a 64-bit
        // division per record, one proton's 1000 recorded steps took 906 us, counting 803)
        const int nsteps = (int)P.nsteps;
        const int rec_every = P.rec_every > 0x7fffffff ? 0x7fffffff : (int)P.rec_every;
        const int64_t until64 = P.rec_every - 1 - (P.step0 % P.rec_every);
        int until = until64 > 0x7fffffff ? 0x7fffffff : (int)until64;   // beyond this launch anyway
        int64_t rec = P.step0 / P.rec_every + 1;
        auto record = [&](V3 rr, V3 vv) {
            if (P.r_hist) {
                write_row(row_at(P.r_hist, rec, n, row), rr);
                write_row(row_at(P.v_hist, rec, n, row), vv);
            }
            ++rec;
        };
        // record-free segments: the inner loop carries only its counter
        int k = 0;
        int quiet = 0;   // upcoming steps known to be field-free (quiet_steps_f64)
        ClearBox clear;
        if constexpr (COLL) clear = no_clear_box();
        while (k < nsteps) {
            const unsigned to_rec = (unsigned)until + 1u;
            const int seg = (int)(to_rec < (unsigned)(nsteps - k) ? to_rec : (unsigned)(nsteps - k));
            const int64_t g0 = P.step0 + k;
            if constexpr (COLL) {
                // each segment is tested unless it ends in the clear box it starts in;
                // a field-free run takes the steps that stay in it
                int i = 0;
                while (i < seg) {
                    if constexpr (alg_skips_free(ALG)) {
                        if (quiet > 0) {
                            const V3 u = state_velocity<ALG>(w, vel);
                            int m = clear_steps(clear, r, P.dt * u);
                            m = min(m, min(quiet, seg - i));
                            if (m > 0) {
                                r = drift_run(r, u, P.dt, m);
                                i += m;
                                quiet -= m;
                                continue;
                            }
                        }
                    }
                    const V3 r0 = r;
                    const bool free = step<ALG, RF, L>(c, r, w, vel, g0 + i, K);
                    ++i;
                    if (!in_clear_box(clear, r)) {
                        if (segment_hits_surface(P.surf, r0, r)) {
                            stopped = true;
                            break;
                        }
                        clear = clear_box(P.surf, r);
                    }
                    if constexpr (alg_skips_free(ALG)) {
                        if (quiet > 0) --quiet;
                        else if (free) quiet = quiet_steps_f64(P.F, r, state_velocity<ALG>(w, vel), P.dt);
                    }
                }
                k += i;
                // the reference records the step's position before its collision test
                if ((unsigned)i == to_rec) {
                    record(r, state_velocity<ALG>(w, vel));
                    until = rec_every - 1;
                } else {
                    until -= i;
                }
                if (stopped) break;
                continue;
            }
            if constexpr (alg_skips_free(ALG)) {
                for (int i = 0; i < seg;) {
                    if (quiet > 0) {
                        // a run of field-free steps: the same position advance, no field lookups
                        const int m = quiet < seg - i ? quiet : seg - i;
                        r = drift_run(r, state_velocity<ALG>(w, vel), P.dt, m);
                        i += m;
                        quiet -= m;
                    } else {
                        if (step<ALG, RF, L>(c, r, w, vel, g0 + i, K))
                            quiet = quiet_steps_f64(P.F, r, state_velocity<ALG>(w, vel), P.dt);
                        ++i;
                    }
                }
            } else {
                for (int i = 0; i < seg; ++i) step<ALG, RF, L>(c, r, w, vel, g0 + i, K);
            }
            k += seg;
            if ((unsigned)seg == to_rec) {
                record(r, state_velocity<ALG>(w, vel));
                until = rec_every - 1;
            } else {
                until -= seg;
            }
        }
        if ((P.flags & PPT_TRACK_FINAL) && !stopped) {
            if constexpr (alg_staggered(ALG)) {
                V3 E, B;
                fields_at<RF, L>(c, r, P.nsteps_total, 0.0, E, B);
                w = half_kick<ALG, L>(w, E, B, 0.5 * P.dt, P.qm);
                if (P.v_hist) write_row(row_at(P.v_hist, P.n_rec - 1, n, row), w_to_v<ALG>(w));
            }
        }
        st[s] = r.x;
        st[n + s] = r.y;
        st[2 * n + s] = r.z;
        st[3 * n + s] = w.x;
        st[4 * n + s] = w.y;
        st[5 * n + s] = w.z;
        if (P.status) {
            double sum = r.x + r.y + r.z + w.x + w.y + w.z;
            if (!isfinite(sum)) atomicOr(P.status, PPT_STATUS_NONFINITE);
        }
        if constexpr (COLL) {
            if (stopped) {
                P.active[row] = 0;
                return (unsigned)k;
            }
        }
    }
    return (unsigned)P.nsteps;
}

// Blocks of 128 per SM the launch bounds ask for (small bunches, resident with
// any of them, gain 1-8 % from no bound: not worth a second set of kernels): the Boris family's kernels
// of a pruned record layout fit 80 registers without spills (6 blocks: the
// RF-gap map crossing 65.0 -> 62.9 ms against 96 registers and 5 blocks);
// the run-time dispatch and the full record would spill there and keep 5 (with
// the collision test too: 8.3 / 7.5 / 7.2 ms with 4 / 5 / 6 blocks, 1e6 protons x
// 1000 steps in a pipe).  The kernels that keep their corners: 4 blocks of RK4, 5 of
// Vay (1e6 electrons x 200 rk4_rel steps, {Ex Ey Bz}: no bound 9.85 ms, 3 / 4 /
// 5 blocks 7.70 / 6.99 / 8.03; 4e5 x 500 vay_rel steps 4 / 5 / 6 blocks 3.06 /
// 2.87 / 3.56), one more for the one-element record (ring, 5e5 x 100 rk4_rel
// steps 1.38 -> 1.34 ms, vay_rel 0.644 -> 0.600).
__host__ __device__ constexpr int f64_min_blocks(int alg, bool coll, int layout) {
    if (keeps_corners(alg, layout) && !coll) {
        const int narrow = layout_width(layout) == 1 ? 1 : 0;
        return ((alg == PPT_ALG_RK4 || alg == PPT_ALG_RK4_REL) ? 4 : 5) + narrow;
    }
    return !alg_skips_free(alg) ? 1 : (layout != 0 && layout != kLayFull) ? 6 : 5;
}

// L = 0: any fields; L = a kLay* mask: one uniform-grid map of that record
// layout, no constant parts (fields_at, boris_v_m).
template <int ALG, bool RF, bool COLL, int L>
__global__ void __launch_bounds__(128, f64_min_blocks(ALG, COLL, L)) track_f64_kernel(const __grid_constant__ TrackDev P) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned steps_done = 0;
    Ctx c = make_ctx(P);
    if constexpr (RF) {
        extern __shared__ double2 rf_tab64[];
        if (P.rf_tab_n > 0) {
            build_rf_table64(rf_tab64, P.step0, P.rf_tab_n, P.omega * P.dt);
            c.tab = rf_tab64;
            c.tab0 = P.step0;
        }
    }
    if (s < P.n) steps_done = track_f64_particle<ALG, RF, COLL, L>(P, s, c);
    if (P.counters) block_add_counters(P.counters, c.hits, steps_done);
}

// Serving: a persistent block-level work queue over the float64 jobs of one
// (algorithm, RF) class.  Each item is one job's 128-particle block; the job's
// parameter block is staged in shared memory and its step window for this
// tick comes from the device-resident step counters.
static_assert(sizeof(TrackDev) % 8 == 0, "TrackDev is copied as 8-byte words");

template <int ALG, bool RF, int L>
__global__ void __launch_bounds__(kJobBlock) track_f64_jobs_kernel(const __grid_constant__ JobQueueDev Q) {
    __shared__ __align__(16) TrackDev sP;
    __shared__ int s_item, s_job;
    const TrackDev* table = static_cast<const TrackDev*>(Q.table);
    for (;;) {
        take_item(Q, &s_item, &s_job);
        const int it = s_item;
        if (it >= Q.n_items) return;
        const int cj = s_job;
        const int gjob = Q.job_index[cj];
        {
            const uint64_t* src = reinterpret_cast<const uint64_t*>(table + Q.table_index[cj]);
            uint64_t* dst = reinterpret_cast<uint64_t*>(&sP);
            for (int i = threadIdx.x; i < (int)(sizeof(TrackDev) / 8); i += blockDim.x) dst[i] = src[i];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int64_t s0, k;
            int fl;
            job_window(Q, gjob, sP.nsteps_total, &s0, &k, &fl);
            sP.step0 = s0;
            sP.nsteps = k;
            sP.flags = Q.done[gjob] ? -1 : fl;   // -1: job finished, nothing to do
        }
        __syncthreads();
        if (sP.flags >= 0) {
            const int64_t s = (int64_t)(it - Q.item_start[cj]) * blockDim.x + threadIdx.x;
            Ctx c = make_ctx(sP);
            unsigned sd = 0;
            if (s < sP.n) sd = track_f64_particle<ALG, RF, false, L>(sP, s, c);
            if (sP.counters) block_add_counters(sP.counters, c.hits, sd);
        }
        __syncthreads();
    }
}

}  // namespace ppt
