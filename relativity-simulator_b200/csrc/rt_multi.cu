// rt_multi.cu -- multi-source Kerr-Schild tracer for sm_100a (FP64).
//
// SoftwareComputeEngine's multi-source path (software_compute_engine.hpp:
// 2708-3252): the camera's hole at the origin plus black-hole bodies, each with
// its own mass, spin axis and thin disk.  The ray equations sum every source's
// Kerr-Schild terms evaluated in that source's local frame (ms_rhs :2857-2871);
// they are the Hamiltonian flow of H = (|p|^2 - 1)/2 - sum_i H_i s_i^2
// (s_i = 1 + k_i . p), onto whose zero set each accepted step is projected.
// The reference steps this path with heuristic RK4; here it runs under the
// DP45 + PI30 machinery of the single-hole tracer, with
//   - a step cap from the nearest source, |h| <= c min_i max(r_i - r_+i, 0.01 m_i);
//   - capture inside capture_scale * r_+ of any source, or when |p| exceeds
//     1000 (a horizon-like region of the summed fields, flag DIVERGED);
//   - escape at |x| > escape radius, the terminal point interpolated to it;
//   - a disk hit at the earliest local-equator crossing of a step that lies on
//     that source's disk, solved on the step's 4th-order dense output, with
//     g = redshift_at(m_i, a_i, r, L_z), L_z from the unit local momentum as in
//     trace_multi_source (:3155).
// Sources live in global memory per bundle (at most 16, read through L1 by
// whole warps of one bundle).  The stage loop is rolled around one copy of the
// N-source RHS, its stage derivatives in shared memory.  In launches of few rays
// several lanes share a ray (Group).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "rt_device.cuh"
#include "rt_internal.h"

namespace relsim {

namespace {

constexpr double kMsMaxMomentum = 1e3;
constexpr double kTwoPi = 6.283185307179586476925286766559;
enum MsMode : int { MS_IDLE = 0, MS_STEP = 1 };

// Dormand-Prince rows for the rolled step (rk45_adaptive.hpp:196-203): row s
// gives the weights of k1..k(s+1) in the input of stage s + 2; row 5 is the
// 5th-order solution.  kMsE: error weights of k1..k7.
__constant__ double kMsA[6][6] = {
    {DP::A21, 0, 0, 0, 0, 0},
    {DP::A31, DP::A32, 0, 0, 0, 0},
    {DP::A41, DP::A42, DP::A43, 0, 0, 0},
    {DP::A51, DP::A52, DP::A53, DP::A54, 0, 0},
    {DP::A61, DP::A62, DP::A63, DP::A64, DP::A65, 0},
    {DP::B1, 0.0, DP::B3, DP::B4, DP::B5, DP::B6}};
__constant__ double kMsE[7] = {DP::E1, 0.0, DP::E3, DP::E4, DP::E5, DP::E6, DP::E7};
__constant__ double kMsD[7] = {DP::D1, 0.0, DP::D3, DP::D4, DP::D5, DP::D6, DP::D7};

template <int BLOCK>
struct MsCold {
    double k[6][6][BLOCK];  // stage derivatives k2..k7
    double lambda[BLOCK];
    double dH[BLOCK];
    double phi[BLOCK];
    uint64_t local[BLOCK];
};

__device__ __forceinline__ double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// ---- the superposed right-hand side ----
//
// A source's term is a chain of some 60 dependent FP64 operations, and a ray takes six
// of them per source and attempt in turn: latency bounds the kernel, not the FP64
// pipe.  Two ways to overlap terms: one lane interleaves U sources, or G lanes of a
// warp share a ray, each evaluating every G-th source.  The terms are always added up
// in source order, and every product and sum is written with its rounding (no
// contraction is left to the compiler), so a ray's steps depend on neither G nor U.
template <int G>
struct Group {
    unsigned mask;  // the group's lanes
    int sub;        // this lane's place among them
    __device__ __forceinline__ double from(double v, int q) const {
        if constexpr (G == 1) return v;
        else return __shfl_sync(mask, v, q, G);
    }
};

// a . b, the first product fused into the second
__device__ __forceinline__ double dot3x(const double* a, const double* b) {
    return __fma_rn(a[2], b[2], __fma_rn(a[0], b[0], __dmul_rn(a[1], b[1])));
}

// Component k in the world frame of a vector with local components v.
__device__ __forceinline__ double ms_world(const MsSource& s, const double* v, int k) {
    return __fma_rn(v[2], s.axis[k], __fma_rn(v[0], s.fx[k], __dmul_rn(v[1], s.fy[k])));
}

// r^2 of a local Kerr-Schild point and the pieces that share it.
template <bool FAST>
__device__ __forceinline__ double ms_r2(const double* x, double a2, double z2, bool square_fused) {
    double d = __fma_rn(x[0], x[0], __dmul_rn(x[1], x[1]));
    d = __dadd_rn(__dadd_rn(d, z2), -a2);
    const double t4 = __dmul_rn(4.0, a2);
    const double v = square_fused ? __fma_rn(d, d, __dmul_rn(t4, z2)) : __fma_rn(t4, z2, __dmul_rn(d, d));
    if constexpr (FAST) {
        const double r2 = __dmul_rn(0.5, __dadd_rn(d, fast_sqrt(v)));
        return (r2 < 1e-24) ? 1e-24 : r2;
    } else {
        return fmax(__dmul_rn(0.5, __dadd_rn(d, __dsqrt_rn(v))), 1e-24);
    }
}

// U sources' terms of the right-hand side in the world frame (the gravitational part
// of ks_rhs in each local frame), with r_BL in that frame.  The reciprocal roots sit
// between two straight-line halves, each of which interleaves the sources.
template <int U, bool FAST>
__device__ __forceinline__ void ms_terms(const MsSource* __restrict__ const* sp, const double* __restrict__ y,
                                         double (*__restrict__ term)[6], double* __restrict__ rout) {
    double X[U][3], P[U][3], R2[U], IR[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const MsSource& s = *sp[u];
        const double rel[3] = {__dadd_rn(y[0], -s.pos[0]), __dadd_rn(y[1], -s.pos[1]), __dadd_rn(y[2], -s.pos[2])};
        X[u][0] = dot3x(rel, s.fx);
        X[u][1] = dot3x(rel, s.fy);
        X[u][2] = dot3x(rel, s.axis);
        P[u][0] = dot3x(y + 3, s.fx);
        P[u][1] = dot3x(y + 3, s.fy);
        P[u][2] = dot3x(y + 3, s.axis);
        R2[u] = ms_r2<FAST>(X[u], __dmul_rn(s.a, s.a), __dmul_rn(X[u][2], X[u][2]), true);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) IR[u] = rsqrt(R2[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const MsSource& s = *sp[u];
        const double* x = X[u];
        const double px = P[u][0], py = P[u][1], pz = P[u][2];
        const double M = FAST ? s.m_fast : s.m, a = s.a;
        const double a2 = __dmul_rn(a, a), z2 = __dmul_rn(x[2], x[2]);
        const double r2 = R2[u], inv_r = IR[u];
        const double r = __dmul_rn(r2, inv_r);
        const double rpa = __dadd_rn(r2, a2);
        const double r4 = __dmul_rn(r2, r2);
        const double den = __fma_rn(a2, z2, r4);
        double q;
        if constexpr (FAST) q = fast_rcp(__dmul_rn(rpa, den));
        else q = __drcp_rn(__dmul_rn(rpa, den));
        const double inv_rpa = __dmul_rn(den, q), inv_den = __dmul_rn(rpa, q);
        const double r3 = __dmul_rn(r2, r);
        const double H = __dmul_rn(__dmul_rn(M, r3), inv_den);
        const double k[3] = {__dmul_rn(__fma_rn(a, x[1], __dmul_rn(r, x[0])), inv_rpa),
                             __dmul_rn(__fma_rn(r, x[1], -__dmul_rn(a, x[0])), inv_rpa), __dmul_rn(x[2], inv_r)};
        const double sv = __fma_rn(k[2], pz, __fma_rn(k[1], py, __fma_rn(k[0], px, 1.0)));
        const double th = __dmul_rn(__dmul_rn(2.0, H), sv);
        const double r3d = __dmul_rn(r3, inv_den);
        const double drz = __dmul_rn(__dmul_rn(__dmul_rn(r, rpa), x[2]), inv_den);
        const double c = __fma_rn(__dmul_rn(3.0, a2), z2, -r4);
        const double C = __dmul_rn(__dmul_rn(__dmul_rn(M, r2), inv_den), __dmul_rn(c, inv_den));
        const double D = __dmul_rn(__dmul_rn(-2.0, H), __dmul_rn(__dmul_rn(a2, x[2]), inv_den));
        const double tr = __dmul_rn(2.0, r);
        const double w0 = __fma_rn(-tr, k[0], x[0]), w1 = __fma_rn(-tr, k[1], x[1]);
        const double W = __fma_rn(w0, px, __dmul_rn(w1, py));
        const double A = __fma_rn(inv_rpa, W, -__dmul_rn(__dmul_rn(inv_r, k[2]), pz));
        const double B0 = __dmul_rn(inv_rpa, __fma_rn(r, px, -__dmul_rn(a, py)));
        const double B1 = __dmul_rn(inv_rpa, __fma_rn(a, px, __dmul_rn(r, py)));
        const double B2 = __dmul_rn(inv_r, pz);
        const double s2 = __dmul_rn(sv, sv);
        const double Gd = __fma_rn(s2, C, __dmul_rn(th, A));
        const double dx[3] = {-__dmul_rn(th, k[0]), -__dmul_rn(th, k[1]), -__dmul_rn(th, k[2])};
        const double dp[3] = {__fma_rn(th, B0, __dmul_rn(__dmul_rn(r3d, x[0]), Gd)),
                              __fma_rn(th, B1, __dmul_rn(__dmul_rn(r3d, x[1]), Gd)),
                              __fma_rn(s2, D, __fma_rn(th, B2, __dmul_rn(drz, Gd)))};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            term[u][i] = ms_world(s, dx, i);
            term[u][3 + i] = ms_world(s, dp, i);
        }
        rout[u] = r;
    }
}

// Superposed RHS; returns min_i max(r_i - r_+i, 0.01 m_i) and the first source
// whose local r_BL < capture_scale r_+ (-1: none).
template <int G, int U, bool FAST>
__device__ __forceinline__ double ms_rhs(const MsSource* __restrict__ src, uint32_t n, const double* __restrict__ y,
                                         double* __restrict__ dy, double cap_scale, int& inside, const Group<G>& grp) {
    double cap = 1e300;
    int in = 0x7fffffff;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        dy[k] = y[3 + k];
        dy[3 + k] = 0.0;
    }
    uint32_t base = 0;
    if constexpr (U > 1) {
#pragma unroll 1
        for (; base + U <= n; base += U) {
            double term[U][6], r[U];
            const MsSource* sp[U];
#pragma unroll
            for (int u = 0; u < U; ++u) sp[u] = src + base + u;
            ms_terms<U, FAST>(sp, y, term, r);
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int k = 0; k < 6; ++k) dy[k] = __dadd_rn(dy[k], term[u][k]);
                cap = fmin(cap, fmax(r[u] - sp[u]->rh, 0.01 * (FAST ? sp[u]->m_fast : sp[u]->m)));
                if (r[u] < cap_scale * sp[u]->rh && in == 0x7fffffff) in = static_cast<int>(base + u);
            }
        }
    }
#pragma unroll 1
    for (; base < n; base += G) {
        double term[1][6], r[1];
        const uint32_t i = base + grp.sub;
        if (i < n) {
            const MsSource* sp[1] = {src + i};
            ms_terms<1, FAST>(sp, y, term, r);
            cap = fmin(cap, fmax(r[0] - sp[0]->rh, 0.01 * (FAST ? sp[0]->m_fast : sp[0]->m)));
            if (r[0] < cap_scale * sp[0]->rh && in == 0x7fffffff) in = static_cast<int>(i);
        } else {
#pragma unroll
            for (int k = 0; k < 6; ++k) term[0][k] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            double t[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) t[k] = grp.from(term[0][k], q);
            if (base + q < n) {
#pragma unroll
                for (int k = 0; k < 6; ++k) dy[k] = __dadd_rn(dy[k], t[k]);
            }
        }
    }
    if constexpr (G > 1) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            cap = fmin(cap, __shfl_xor_sync(grp.mask, cap, o, G));
            in = min(in, __shfl_xor_sync(grp.mask, in, o, G));
        }
    }
    inside = (in == 0x7fffffff) ? -1 : in;
    return cap;
}

// Stages 2..7 around one RHS copy; K holds k2..k7 on return.  The stage sums are
// unrolled over j (predicated), so their shared-memory loads issue together.
template <int BLOCK, int G, int U, bool FAST>
__device__ __forceinline__ void ms_stages(const MsSource* __restrict__ src, uint32_t n, const double* __restrict__ y,
                                          const double* __restrict__ k1, double hh, MsCold<BLOCK>& S, int tid,
                                          double cap_scale, double* __restrict__ y5, double* __restrict__ k7,
                                          double* __restrict__ est, double& cap5, int& inside5, const Group<G>& grp) {
#pragma unroll 1
    for (int st = 0; st < 6; ++st) {
        double in[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double acc = __dmul_rn(kMsA[st][0], k1[i]);
#pragma unroll
            for (int j = 1; j < 6; ++j)
                if (j <= st) acc = __fma_rn(kMsA[st][j], S.k[j - 1][i][tid], acc);
            in[i] = __fma_rn(hh, acc, y[i]);
        }
        if (st == 5) {
#pragma unroll
            for (int i = 0; i < 6; ++i) y5[i] = in[i];
        }
        double out[6];
        int ins;
        const double c = ms_rhs<G, U, FAST>(src, n, in, out, cap_scale, ins, grp);
#pragma unroll
        for (int i = 0; i < 6; ++i) S.k[st][i][tid] = out[i];
        if (st == 5) {
#pragma unroll
            for (int i = 0; i < 6; ++i) k7[i] = out[i];
            cap5 = c;
            inside5 = ins;
        }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        double acc = __dmul_rn(kMsE[0], k1[i]);
#pragma unroll
        for (int j = 2; j < 7; ++j) acc = __fma_rn(kMsE[j], S.k[j - 1][i][tid], acc);
        est[i] = __dmul_rn(fabs(hh), fabs(acc));
    }
}

// The attempt with the compiler's division and root, for an attempt whose stages
// leave the fast forms' range (its error estimate is NaN: one NaN term makes all six
// sums NaN).  Out of line: y and k1 in io[0..11], then y5, k7, est and cap5.
template <int BLOCK, int G>
__device__ __noinline__ int ms_stages_special(const MsSource* __restrict__ src, uint32_t n, double* __restrict__ io,
                                              double hh, MsCold<BLOCK>& S, int tid, double cap_scale,
                                              const Group<G> grp) {
    double y[6], k1[6], y5[6], k7[6], est[6], cap5 = 0.0;
    int inside5 = -1;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        y[i] = io[i];
        k1[i] = io[6 + i];
    }
    ms_stages<BLOCK, G, 1, false>(src, n, y, k1, hh, S, tid, cap_scale, y5, k7, est, cap5, inside5, grp);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        io[12 + i] = y5[i];
        io[18 + i] = k7[i];
        io[24 + i] = est[i];
    }
    io[30] = cap5;
    return inside5;
}

// Coefficients of the step's dense output y(t) = y0 + t (d + (1-t)(b + t(c + (1-t) e))).
template <int BLOCK>
__device__ __forceinline__ void ms_dense_coeffs(const double* __restrict__ y0, const double* __restrict__ y1,
                                                const double* __restrict__ k1, const double* __restrict__ k7, double h,
                                                const MsCold<BLOCK>& S, int tid, double (*co)[6]) {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double d = y1[i] - y0[i];
        const double b = h * k1[i] - d;
        double e = kMsD[0] * k1[i] + kMsD[6] * k7[i];
#pragma unroll 1
        for (int j = 2; j < 6; ++j) e += kMsD[j] * S.k[j - 1][i][tid];
        co[0][i] = d;
        co[1][i] = b;
        co[2][i] = d - h * k7[i] - b;
        co[3][i] = h * e;
    }
}

__device__ __forceinline__ double ms_dense_at(const double* y0, const double (*co)[6], int i, double t) {
    return y0[i] + t * (co[0][i] + (1.0 - t) * (co[1][i] + t * (co[2][i] + (1.0 - t) * co[3][i])));
}

// Illinois root on [0, 1] of the local z of source s on the dense output.
__device__ double ms_local_z_root(const MsSource& s, const double* y0, const double (*co)[6], double f0, double f1) {
    double lo = 0.0, hi = 1.0, flo = f0, fhi = f1, t = 1.0;
    int side = 0;
    for (int it = 0; it < 60; ++it) {
        t = (lo * fhi - hi * flo) / (fhi - flo);
        if (!(t > lo && t < hi)) t = 0.5 * (lo + hi);
        const double rel[3] = {ms_dense_at(y0, co, 0, t) - s.pos[0], ms_dense_at(y0, co, 1, t) - s.pos[1],
                               ms_dense_at(y0, co, 2, t) - s.pos[2]};
        const double ft = dot3(rel, s.axis);
        if (ft == 0.0 || fabs(hi - lo) < 1e-15 || fabs(ft) < 1e-13 * (1.0 + fabs(rel[0]) + fabs(rel[1]))) break;
        if ((ft > 0.0) == (fhi > 0.0)) {
            hi = t;
            fhi = ft;
            if (side == -1) flo *= 0.5;
            side = -1;
        } else {
            lo = t;
            flo = ft;
            if (side == 1) fhi *= 0.5;
            side = 1;
        }
    }
    return t;
}

// Fraction of the step where |x| of the cubic Hermite interpolant crosses target.
__device__ double ms_radius_crossing(const double* y0, const double* f0, const double* y1, const double* f1, double h,
                                     double target) {
    double lo = 0.0, hi = 1.0, x[6];
    double flo = sqrt(dot3(y0, y0)) - target, fhi = sqrt(dot3(y1, y1)) - target;
    if (!((flo > 0.0) != (fhi > 0.0))) return 1.0;
    int side = 0;
    double t = 1.0;
    for (int it = 0; it < 60; ++it) {
        t = (lo * fhi - hi * flo) / (fhi - flo);
        if (!(t > lo && t < hi)) t = 0.5 * (lo + hi);
        hermite(y0, f0, y1, f1, h, t, 3, x);
        const double ft = sqrt(dot3(x, x)) - target;
        if (ft == 0.0 || fabs(hi - lo) < 1e-15 || fabs(ft) < 1e-13 * target) break;
        if ((ft > 0.0) == (fhi > 0.0)) {
            hi = t;
            fhi = ft;
            if (side == -1) flo *= 0.5;
            side = -1;
        } else {
            lo = t;
            flo = ft;
            if (side == 1) fhi *= 0.5;
            side = 1;
        }
    }
    return t;
}

// Kerr-Schild field of one source at a world point: k in the world frame, H.
template <bool FAST>
__device__ __forceinline__ double ms_field(const MsSource& s, const double* __restrict__ at, double* __restrict__ kw) {
    const double rel[3] = {__dadd_rn(at[0], -s.pos[0]), __dadd_rn(at[1], -s.pos[1]), __dadd_rn(at[2], -s.pos[2])};
    const double x[3] = {dot3x(rel, s.fx), dot3x(rel, s.fy), dot3x(rel, s.axis)};
    const double a = s.a, a2 = __dmul_rn(a, a);
    const double r2 = ms_r2<FAST>(x, a2, __dmul_rn(x[2], x[2]), false);
    const double inv_r = rsqrt(r2);
    const double r = __dmul_rn(r2, inv_r);
    const double rpa = __dadd_rn(r2, a2);
    const double den = __fma_rn(__dmul_rn(a2, x[2]), x[2], __dmul_rn(r2, r2));
    double q;
    if constexpr (FAST) q = fast_rcp(__dmul_rn(rpa, den));
    else q = __drcp_rn(__dmul_rn(rpa, den));
    const double inv_rpa = __dmul_rn(den, q);
    const double k[3] = {__dmul_rn(__fma_rn(a, x[1], __dmul_rn(r, x[0])), inv_rpa),
                         __dmul_rn(__fma_rn(r, x[1], -__dmul_rn(a, x[0])), inv_rpa), __dmul_rn(x[2], inv_r)};
#pragma unroll
    for (int i = 0; i < 3; ++i) kw[i] = ms_world(s, k, i);
    return __dmul_rn(__dmul_rn(__dmul_rn(FAST ? s.m_fast : s.m, r2), r), __dmul_rn(rpa, q));
}

// Projection of p onto H = 0 along n = dH/dp, closest root; returns |H| before (NaN,
// with p as it was, where a field leaves the fast forms' range).  Two passes over
// the sources (n needs all of them first).
template <int G, bool FAST>
__device__ __forceinline__ double ms_project(const MsSource* __restrict__ src, uint32_t n, double* y, double tol,
                                             const Group<G>& grp) {
    double* p = y + 3;
    double nv[3] = {p[0], p[1], p[2]};
    double sum = 0.0;
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += G) {
        const uint32_t i = base + grp.sub;
        double kw[3] = {0.0, 0.0, 0.0}, hs = 0.0, sv = 0.0, c = 0.0;
        if (i < n) {
            const double hf = ms_field<FAST>(src[i], y, kw);
            sv = __dadd_rn(1.0, dot3x(kw, p));
            hs = __dmul_rn(hf, sv);
            c = __dmul_rn(__dmul_rn(2.0, hf), sv);
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const double hq = grp.from(hs, q), sq = grp.from(sv, q), cq = grp.from(c, q);
            double kq[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) kq[k] = grp.from(kw[k], q);
            if (base + q < n) {
                sum = __fma_rn(hq, sq, sum);
#pragma unroll
                for (int k = 0; k < 3; ++k) nv[k] = __fma_rn(-cq, kq[k], nv[k]);
            }
        }
    }
    const double res = __fma_rn(0.5, __dadd_rn(dot3x(p, p), -1.0), -sum);
    if (!(fabs(res) >= tol)) return fabs(res);
    double qa = __dmul_rn(0.5, dot3x(nv, nv)), qb = dot3x(p, nv);
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += G) {
        const uint32_t i = base + grp.sub;
        double kn = 0.0, ha = 0.0, hb = 0.0;
        if (i < n) {
            double kw[3];
            const double hf = ms_field<FAST>(src[i], y, kw);
            const double sv = __dadd_rn(1.0, dot3x(kw, p));
            kn = dot3x(kw, nv);
            ha = __dmul_rn(hf, kn);
            hb = __dmul_rn(__dmul_rn(2.0, hf), sv);
        }
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const double kq = grp.from(kn, q), aq = grp.from(ha, q), bq = grp.from(hb, q);
            if (base + q < n) {
                qa = __fma_rn(-aq, kq, qa);
                qb = __fma_rn(-bq, kq, qb);
            }
        }
    }
    const double disc = __fma_rn(qb, qb, -__dmul_rn(__dmul_rn(4.0, qa), res));
    if (disc >= 0.0) {
        const double q = __dmul_rn(-0.5, __dadd_rn(qb, copysign(__dsqrt_rn(disc), qb)));
        if (q != 0.0) {
            const double alpha = __ddiv_rn(res, q);
#pragma unroll
            for (int k = 0; k < 3; ++k) p[k] = __fma_rn(alpha, nv[k], p[k]);
        }
    }
    return fabs(res);
}

template <int G>
__device__ __noinline__ double ms_project_special(const MsSource* __restrict__ src, uint32_t n, double* y, double tol,
                                                  const Group<G> grp) {
    return ms_project<G, false>(src, n, y, tol, grp);
}

// Static observer's null momentum in the superposed metric (ms_initial_momentum,
// software_compute_engine.hpp:2915-2964).
__device__ __noinline__ void ms_initial_momentum(const MsSource* __restrict__ src, uint32_t n, const double* x,
                                                 const double* outward, double* pout) {
    // potentials and world directions are recomputed where needed (no per-source arrays)
    auto field = [&](uint32_t i, double& pot, double* dir) {
        const MsSource& s = src[i];
        const double rel[3] = {x[0] - s.pos[0], x[1] - s.pos[1], x[2] - s.pos[2]};
        const double lx[3] = {dot3(rel, s.fx), dot3(rel, s.fy), dot3(rel, s.axis)};
        double kl[3];
        ks_field64(lx, s.m, s.a, kl, pot);
#pragma unroll
        for (int k = 0; k < 3; ++k) dir[k] = kl[0] * s.fx[k] + kl[1] * s.fy[k] + kl[2] * s.axis[k];
    };
    auto mdot = [&](const double* a, const double* b) {
        double v = -a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3];
        for (uint32_t i = 0; i < n; ++i) {
            double pot, dir[3];
            field(i, pot, dir);
            const double la = a[0] + dir[0] * a[1] + dir[1] * a[2] + dir[2] * a[3];
            const double lb = b[0] + dir[0] * b[1] + dir[1] * b[2] + dir[2] * b[3];
            v += 2.0 * pot * la * lb;
        }
        return v;
    };
    double sum = 0.0;
    double e[3][4];
    for (int j = 0; j < 3; ++j) e[j][0] = 0.0;
    for (uint32_t i = 0; i < n; ++i) {
        double pot, dir[3];
        field(i, pot, dir);
        sum += pot;
        for (int j = 0; j < 3; ++j) e[j][0] += pot * dir[j];  // shift of axis j
    }
    const double ilsq = 1.0 / fmax(1.0 - 2.0 * sum, 1e-6);
    const double u0 = sqrt(ilsq);
    for (int j = 0; j < 3; ++j) {
        e[j][0] = 2.0 * e[j][0] * ilsq;
        e[j][1] = (j == 0) ? 1.0 : 0.0;
        e[j][2] = (j == 1) ? 1.0 : 0.0;
        e[j][3] = (j == 2) ? 1.0 : 0.0;
    }
    for (int j = 0; j < 3; ++j) {
        double d[2] = {0.0, 0.0};
        for (int q = 0; q < j; ++q) d[q] = mdot(e[j], e[q]);
        for (int q = 0; q < j; ++q)
            for (int c = 0; c < 4; ++c) e[j][c] -= d[q] * e[q][c];
        const double norm = sqrt(fmax(mdot(e[j], e[j]), 1e-30));
        for (int c = 0; c < 4; ++c) e[j][c] /= norm;
    }
    double v[4];
    for (int c = 0; c < 4; ++c) v[c] = -outward[0] * e[0][c] - outward[1] * e[1][c] - outward[2] * e[2][c];
    v[0] += u0;
    double mom[3] = {v[1], v[2], v[3]};
    double tc = -v[0];
    for (uint32_t i = 0; i < n; ++i) {
        double pot, dir[3];
        field(i, pot, dir);
        const double lv = v[0] + dir[0] * v[1] + dir[1] * v[2] + dir[2] * v[3];
        tc += 2.0 * pot * lv;
        for (int k = 0; k < 3; ++k) mom[k] += 2.0 * pot * lv * dir[k];
    }
    const double inv = 1.0 / fmax(-tc, 1e-12);
    for (int k = 0; k < 3; ++k) pout[k] = mom[k] * inv;
}

// Ray generation: pixel -> pinhole direction -> world direction (as the
// single-hole tracer), the observer's Cartesian point, initial momentum.
__device__ __noinline__ void ms_init_ray(const MsDesc* __restrict__ Bp, const MsSource* __restrict__ src,
                                         uint64_t local, double* __restrict__ y) {
    const MsDesc& B = *Bp;
    const uint32_t row = static_cast<uint32_t>(local / B.ncols);
    const uint32_t col = static_cast<uint32_t>(local - static_cast<uint64_t>(row) * B.ncols);
    const double px = static_cast<double>(B.col0 + col);
    const double py = static_cast<double>(B.row0 + row);
    const double v = 1.0 - (py + 0.5) / static_cast<double>(B.height) * 2.0;
    const double u = ((px + 0.5) / static_cast<double>(B.width) * 2.0 - 1.0) * B.aspect;
    const double n2 = v * B.tan_half_fov, n3 = u * B.tan_half_fov;
    const double len = sqrt(1.0 + n2 * n2 + n3 * n3);
    const double inv = (len > 0.0) ? (1.0 / len) : 1.0;
    const double nl0 = inv, nl1 = n2 * inv, nl2 = n3 * inv;
    double d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = nl0 * B.fwd[i] + nl2 * B.rgt[i] + nl1 * B.up[i];
    y[0] = B.x0[0];
    y[1] = B.x0[1];
    y[2] = B.x0[2];
    ms_initial_momentum(src, B.src_count, y, d, y + 3);
}

template <int BLOCK>
__device__ __noinline__ void ms_finish(const MsDesc* __restrict__ Bp, const MsSource* __restrict__ src,
                                       MsCold<BLOCK>& S, int tid, const double* y,
                                       uint32_t status, uint32_t flags, uint32_t acc, uint32_t rej, double r_hit,
                                       double g, uint32_t body, const OutPtrs& out) {
    const double r = sqrt(dot3(y, y));
    const double theta = acos(fmin(fmax(y[2] / fmax(r, 1e-300), -1.0), 1.0));
    const uint64_t o = Bp->out_offset + S.local[tid];
    const rt_ray_out& R = out.rays;
    if (R.status) R.status[o] = status;
    if (R.flags) R.flags[o] = flags;
    if (R.steps_accepted) R.steps_accepted[o] = acc;
    if (R.steps_rejected) R.steps_rejected[o] = rej;
    if (R.r) R.r[o] = r;
    if (R.theta) R.theta[o] = theta;
    if (R.phi) R.phi[o] = S.phi[tid];
    if (R.r_hit) R.r_hit[o] = r_hit;
    if (R.g) R.g[o] = g;
    if (R.lambda) R.lambda[o] = S.lambda[tid];
    if (R.dH) R.dH[o] = S.dH[tid];
    if (R.dE) R.dE[o] = NAN;
    if (R.dLz) R.dLz[o] = NAN;
    if (R.dQ) R.dQ[o] = NAN;
    if (R.body) R.body[o] = body;
    if (R.exit_x || R.exit_y || R.exit_z) {
        // sky-lookup direction of an escaped ray: minus the normalised flow of the
        // superposed RHS at the terminal state, (0, 0, -1) where it vanishes
        // (software_compute_engine.hpp:3220-3224)
        double e[3] = {NAN, NAN, NAN};
        if (status == RT_RAY_ESCAPED) {
            double dy[6];
            int ins;
            ms_rhs<1, 1, false>(src, Bp->src_count, y, dy, Bp->capture_scale, ins, Group<1>{0u, 0});
            const double len = sqrt(dot3(dy, dy));
            if (len > 1e-12) {
#pragma unroll
                for (int i = 0; i < 3; ++i) e[i] = -dy[i] / len;
            } else {
                e[0] = e[1] = 0.0;
                e[2] = -1.0;
            }
        }
        if (R.exit_x) R.exit_x[o] = e[0];
        if (R.exit_y) R.exit_y[o] = e[1];
        if (R.exit_z) R.exit_z[o] = e[2];
    }
    if (out.pixels) {
        const uint32_t pflags = (status == RT_RAY_CAPTURED)  ? RT_PIXEL_HORIZON_ABSORBED
                                : (status == RT_RAY_ESCAPED) ? RT_PIXEL_CELESTIAL_HIT
                                : (status == RT_RAY_DISK)    ? RT_PIXEL_ACCRETION_DISK_HIT
                                                             : 0u;
        float4* p4 = reinterpret_cast<float4*>(out.pixels + o);
        p4[0] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        reinterpret_cast<uint4*>(p4)[1] = make_uint4(__float_as_uint(static_cast<float>(g)),
                                                     __float_as_uint(static_cast<float>(-S.lambda[tid])), pflags, acc);
    }
}

// Translucent-disk continuation of a multi-source ray (trace_multi_source,
// software_compute_engine.hpp:3150-3191): every disk crossing recorded in
// order along the ray (radius, local azimuth, g and the source), the ray
// followed to its end.  End record: crossings, class at the end, and whether
// the end point lies within 6 m of a source (where the reference drops the
// remaining throughput instead of adding the sky, :3207-3216).
__device__ __forceinline__ void ms_cont_record(const ContOut& C, uint64_t o, uint32_t k, double r, double az,
                                               double g) {
    C.cross[(3 * k) * C.stride + o] = r;
    C.cross[(3 * k + 1) * C.stride + o] = az;
    C.cross[(3 * k + 2) * C.stride + o] = g;
}

__device__ __noinline__ void ms_cont_finish(const ContOut& C, uint64_t o, uint32_t n_cross, uint32_t bodies,
                                            uint32_t status, const MsSource* __restrict__ src, uint32_t n,
                                            const double* x) {
    bool near = false;
    for (uint32_t i = 0; i < n; ++i) {
        const double d[3] = {x[0] - src[i].pos[0], x[1] - src[i].pos[1], x[2] - src[i].pos[2]};
        near = near || sqrt(dot3(d, d)) < 6.0 * src[i].m;
    }
    C.info[o] = n_cross | (status << CI_FATE_SHIFT) | (near ? CI_INSIDE_3RS : 0u);
    C.body[o] = bodies;
    if (C.exit) {
        // the sky-lookup direction at the end: minus the normalised flow of the
        // superposed RHS, (0, 0, -1) where it vanishes (:3220-3224)
        double dy[6], e[3] = {0.0, 0.0, -1.0};
        int ins;
        ms_rhs<1, 1, false>(src, n, x, dy, 1.0, ins, Group<1>{0u, 0});
        const double len = sqrt(dot3(dy, dy));
        if (len > 1e-12)
            for (int i = 0; i < 3; ++i) e[i] = -dy[i] / len;
        C.exit[o] = e[0];
        C.exit[C.stride + o] = e[1];
        C.exit[2 * C.stride + o] = e[2];
    }
}

__device__ __forceinline__ void ms_unwrap(double& phi, const double* y) {
    double d = atan2(y[1], y[0]) - phi;
    d -= kTwoPi * floor(d / kTwoPi + 0.5);
    phi += d;
}

// Eight warps per SM: at 12 (168 registers) the two interleaved sources spill, and the
// chain of an attempt, which is what bounds this kernel, gets longer (5 holes: 480x270
// 23.9 ms at 12 warps and one source at a time, 20.3 at 8 and two; 160x90 17.8 / 13.0).
template <int BLOCK, bool CONT, int G, int U>
__global__ void __launch_bounds__(BLOCK, 256 / BLOCK) ms_trace_kernel(MsArgs args) {
    __shared__ MsCold<BLOCK> S;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const Group<G> grp{((1u << G) - 1u) << (lane & ~(G - 1)), lane & (G - 1)};
    const bool leader = grp.sub == 0;

    double y[6], k1[6];
    double h = 0.0, cap_len = 0.0;
    float lnp = 0.0f;
    bool has_hist = false;
    int inside = -1;
    uint32_t acc = 0, rej = 0, flags = 0, bidx = 0, guard = 0;
    int mode = MS_IDLE;
    uint32_t n_cross = 0, bodies = 0;  // continuation: crossings so far, their sources
#pragma unroll
    for (int i = 0; i < 6; ++i) y[i] = k1[i] = 0.0;
    bool queue_open = true;
    uint64_t chunk_next = 0, chunk_end = 0;
    uint32_t n_att = 0, n_acc = 0, n_rays = 0;

    for (;;) {
        // refill idle lanes from the warp's chunk, then from a new chunk (one atomic)
        const unsigned idle = __ballot_sync(FULL, mode == MS_IDLE);
        const int n_idle = __popc(idle);
        if ((queue_open || chunk_next < chunk_end) && n_idle > 0 &&
            (n_idle >= static_cast<int>(args.refill_threshold) || n_idle == 32)) {
            const uint64_t avail = chunk_end - chunk_next;
            uint64_t base2 = 0;
            bool got2 = false;
            const int n_want = n_idle / G;  // idle groups: rays to take
            if (avail < static_cast<uint64_t>(n_want) && queue_open) {
                const int leader = __ffs(idle) - 1;
                unsigned long long b = 0;
                if (lane == leader) b = atomicAdd(args.queue, static_cast<unsigned long long>(args.claim));
                b = __shfl_sync(FULL, b, leader);
                if (b >= args.total_rays) {
                    queue_open = false;
                } else {
                    base2 = b;
                    got2 = true;
                    if (b + args.claim >= args.total_rays) queue_open = false;
                }
            }
            const uint64_t used_old = (avail < static_cast<uint64_t>(n_want)) ? avail : n_want;
            if (mode == MS_IDLE) {
                const uint64_t rank = static_cast<uint64_t>(__popc(idle & lt_mask) / G);
                uint64_t rid = ~0ull;
                if (rank < avail) rid = chunk_next + rank;
                else if (got2) rid = base2 + (rank - avail);
                if (rid < args.total_rays) {
                    uint32_t lo = 0, hi = args.n_bundles;
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (args.bundles[mid].ray_begin <= rid) lo = mid; else hi = mid;
                    }
                    bidx = lo;
                    const MsDesc* Bp = args.bundles + lo;
                    const MsSource* src = args.sources + Bp->src_begin;
                    S.local[tid] = rid - Bp->ray_begin;
                    ms_init_ray(Bp, src, S.local[tid], y);
                    int ins;
                    cap_len = ms_rhs<G, 1, false>(src, Bp->src_count, y, k1, Bp->capture_scale, ins, grp);
                    inside = ins;
                    h = -Bp->h0;
                    lnp = 0.0f;
                    has_hist = false;
                    acc = rej = flags = guard = 0;
                    S.lambda[tid] = 0.0;
                    S.dH[tid] = 0.0;
                    S.phi[tid] = Bp->phi0;
                    n_cross = bodies = 0;
                    mode = MS_STEP;
                    if (leader) ++n_rays;
                }
            }
            if (got2) {
                chunk_next = base2 + (static_cast<uint64_t>(n_want) - used_old);
                chunk_end = base2 + args.claim;
                if (chunk_end > args.total_rays) chunk_end = args.total_rays;
            } else {
                chunk_next += used_old;
            }
        }
        if (__ballot_sync(FULL, mode != MS_IDLE) == 0) {
            if (!queue_open && chunk_next >= chunk_end) break;
            continue;
        }
        if (mode == MS_IDLE) continue;

        const MsDesc* Bp = args.bundles + bidx;
        const MsSource* src = args.sources + Bp->src_begin;
        const uint32_t ns = Bp->src_count;
        // the end of a ray: its record (with the continuation only when it crossed
        // no disk: the record describes the first hit) and its continuation end
        auto end_ray = [&](const double* yend, uint32_t status, uint32_t fl, uint32_t body) {
            if (leader && (!CONT || n_cross == 0))
                ms_finish<BLOCK>(Bp, src, S, tid, yend, status, fl, acc, rej, NAN, 1.0, body, args.out);
            if constexpr (CONT) {
                if (leader)
                    ms_cont_finish(args.cont, Bp->out_offset + S.local[tid], n_cross, bodies, status, src, ns, yend);
            }
            mode = MS_IDLE;
        };
        // backstop on loop iterations per ray (one attempt per iteration)
        uint32_t term = 0;
        if (++guard > Bp->max_steps + 64u) {
            flags |= RT_RAYFLAG_MAX_STEPS;
            term = RT_RAY_UNFINISHED + 16;
        } else if (inside >= 0) {
            term = RT_RAY_CAPTURED;
        } else if (dot3(y + 3, y + 3) > kMsMaxMomentum * kMsMaxMomentum) {
            flags |= RT_RAYFLAG_DIVERGED;
            term = RT_RAY_CAPTURED;
        } else if (dot3(y, y) > Bp->r_esc * Bp->r_esc) {
            term = RT_RAY_ESCAPED;
        } else if (acc + rej >= Bp->max_steps) {
            flags |= RT_RAYFLAG_MAX_STEPS;
            term = RT_RAY_UNFINISHED + 16;
        } else {
            const double cap = Bp->cap_c * cap_len;
            if (fabs(h) > cap) h = -cap;
            if (fabs(h) < 1e-8) {
                flags |= RT_RAYFLAG_STEP_UNDERFLOW;
                term = RT_RAY_CAPTURED;
            }
        }
        if (term) {
            const uint32_t cls = term & 15u;
            end_ray(y, cls, flags,
                    (cls == RT_RAY_CAPTURED && inside >= 0) ? static_cast<uint32_t>(inside) : RT_BODY_NONE);
            continue;
        }

        const double hh = h;
        double y5[6], k7[6], est[6], cap5;
        int inside5;
        ms_stages<BLOCK, G, U, true>(src, ns, y, k1, hh, S, tid, Bp->capture_scale, y5, k7, est, cap5, inside5, grp);
        if (est[2] != est[2]) {  // a stage left the fast forms' range (or the state is NaN)
            double io[31];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                io[i] = y[i];
                io[6 + i] = k1[i];
            }
            inside5 = ms_stages_special<BLOCK, G>(src, ns, io, hh, S, tid, Bp->capture_scale, grp);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                y5[i] = io[12 + i];
                k7[i] = io[18 + i];
                est[i] = io[24 + i];
            }
            cap5 = io[30];
        }
        double err;
        {
            double num = 0.0, den = 1.0;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const double sc = Bp->rtol * fmax(fabs(y[i]), fabs(y5[i])) + Bp->atol;
                if (est[i] * den > num * sc) {
                    num = est[i];
                    den = sc;
                }
            }
            err = num / den;
        }
        if (!(err <= 1e300)) err = 1e300;
        if (leader) ++n_att;
        if (err > 1.0) {
            ++rej;
            const float le = __log2f(fmaxf(static_cast<float>(err), 1e-12f));
            const float factor = pi30_factor(le, has_hist ? lnp : le, 4.0f);
            lnp = le;
            has_hist = true;
            h = -fabs(h) * clampd(0.9 * static_cast<double>(factor), 0.1, 0.9);
            continue;
        }
        ++acc;
        if (leader) ++n_acc;
        bool finite = true;
#pragma unroll
        for (int i = 0; i < 6; ++i) finite = finite && isfinite(y5[i]);
        if (!finite) {
            end_ray(y, RT_RAY_CAPTURED, flags | RT_RAYFLAG_NONFINITE, RT_BODY_NONE);
            continue;
        }
        // disk crossings of this step in order along the ray, each the earliest
        // local-equator crossing on a disk after the previous one: the first ends
        // the ray; under the continuation each is recorded and the ray goes on
        {
            bool ended = false;
            double t_prev = -1.0;
#pragma unroll 1
            for (uint32_t pass = 0; pass < ns; ++pass) {
                double best = 2.0, best_r = 0.0, best_lz = 0.0, best_az = 0.0;
                uint32_t best_i = 0;
#pragma unroll 1
                for (uint32_t i = 0; i < ns; ++i) {
                    const MsSource& s = src[i];
                    if (s.disk_in < 0.0) continue;
                    const double r0[3] = {y[0] - s.pos[0], y[1] - s.pos[1], y[2] - s.pos[2]};
                    const double r1[3] = {y5[0] - s.pos[0], y5[1] - s.pos[1], y5[2] - s.pos[2]};
                    const double z0 = dot3(r0, s.axis), z1 = dot3(r1, s.axis);
                    if (!(z0 * z1 <= 0.0) || z0 == z1) continue;
                    const double sl = z0 / (z0 - z1);
                    const double ce[3] = {r0[0] + sl * (r1[0] - r0[0]), r0[1] + sl * (r1[1] - r0[1]),
                                          r0[2] + sl * (r1[2] - r0[2])};
                    const double lxe = dot3(ce, s.fx), lye = dot3(ce, s.fy);
                    const double re = sqrt(fmax(lxe * lxe + lye * lye - s.a * s.a, 0.0));
                    const double margin = 0.05 * re + 0.5 * s.m;
                    if (re < s.disk_in - margin || re > s.disk_out + margin) continue;
                    double co[4][6];
                    ms_dense_coeffs<BLOCK>(y, y5, k1, k7, hh, S, tid, co);
                    const double t = ms_local_z_root(s, y, co, z0, z1);
                    if (!(t < best) || !(t > t_prev)) continue;
                    double yr[6];
#pragma unroll
                    for (int q = 0; q < 6; ++q) yr[q] = ms_dense_at(y, co, q, t);
                    const double rel[3] = {yr[0] - s.pos[0], yr[1] - s.pos[1], yr[2] - s.pos[2]};
                    const double c0 = dot3(rel, s.fx), c1 = dot3(rel, s.fy);
                    const double pl[3] = {dot3(yr + 3, s.fx), dot3(yr + 3, s.fy), dot3(yr + 3, s.axis)};
                    const double rr = sqrt(fmax(c0 * c0 + c1 * c1 - s.a * s.a, 0.0));
                    if (rr < s.disk_in || rr > s.disk_out || rr <= s.rh * 1.02) continue;
                    best = t;
                    best_r = rr;
                    best_i = i;
                    best_lz = (c0 * pl[1] - c1 * pl[0]) / fmax(sqrt(dot3(pl, pl)), 1e-30);
                    // local azimuth of the crossing (ms_disk_crossing, :3037)
                    best_az = atan2(c1, c0) - atan2(s.a, rr);
                }
                if (best > 1.0) break;
                double co[4][6], yr[6];
                ms_dense_coeffs<BLOCK>(y, y5, k1, k7, hh, S, tid, co);
#pragma unroll
                for (int q = 0; q < 6; ++q) yr[q] = ms_dense_at(y, co, q, best);
                const MsSource& s = src[best_i];
                const double g = disk_redshift(s.m, s.a, best_r, best_lz);
                const double lam = S.lambda[tid], ph0 = S.phi[tid];
                if (!CONT || n_cross == 0) {
                    S.lambda[tid] = lam + best * hh;
                    double ph = ph0;
                    ms_unwrap(ph, yr);
                    S.phi[tid] = ph;
                    if (leader) ms_finish<BLOCK>(Bp, src, S, tid, yr, RT_RAY_DISK, flags, acc, rej, best_r, g, best_i, args.out);
                }
                if constexpr (!CONT) {
                    mode = MS_IDLE;
                    ended = true;
                    break;
                } else {
                    // the crossing recorded; the ray goes on through the disk
                    S.lambda[tid] = lam;
                    S.phi[tid] = ph0;
                    if (leader)
                        ms_cont_record(args.cont, Bp->out_offset + S.local[tid], n_cross, best_r, best_az, g);
                    bodies |= best_i << (4u * n_cross);
                    ++n_cross;
                    t_prev = best;
                    if (n_cross >= kMaxCrossings) {
                        if (leader)
                            ms_cont_finish(args.cont, Bp->out_offset + S.local[tid], n_cross, bodies,
                                           RT_RAY_UNFINISHED, src, ns, yr);
                        mode = MS_IDLE;
                        ended = true;
                        break;
                    }
                }
            }
            if (ended) continue;
        }
        if (inside5 >= 0) {  // captured inside this step: its end point
            S.lambda[tid] += hh;
            double ph = S.phi[tid];
            ms_unwrap(ph, y5);
            S.phi[tid] = ph;
            end_ray(y5, RT_RAY_CAPTURED, flags, static_cast<uint32_t>(inside5));
            continue;
        }
        if (dot3(y5, y5) > Bp->r_esc * Bp->r_esc) {  // escaped: interpolated to the escape radius
            const double t = ms_radius_crossing(y, k1, y5, k7, hh, Bp->r_esc);
            double yt[6];
            hermite(y, k1, y5, k7, hh, t, 6, yt);
            S.lambda[tid] += t * hh;
            double ph = S.phi[tid];
            ms_unwrap(ph, yt);
            S.phi[tid] = ph;
            end_ray(yt, RT_RAY_ESCAPED, flags, RT_BODY_NONE);
            continue;
        }
        {
            double drift = ms_project<G, true>(src, ns, y5, Bp->proj_tol, grp);
            if (drift != drift) drift = ms_project_special<G>(src, ns, y5, Bp->proj_tol, grp);
            S.dH[tid] = fmax(S.dH[tid], drift);
        }
        {
            double ph = S.phi[tid];
            ms_unwrap(ph, y5);
            S.phi[tid] = ph;
        }
        S.lambda[tid] += hh;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            y[i] = y5[i];
            k1[i] = k7[i];
        }
        cap_len = cap5;
        inside = inside5;
        float factor = 5.0f;
        if (err != 0.0) {
            const float le = __log2f(fmaxf(static_cast<float>(err), 1e-12f));
            factor = pi30_factor(le, has_hist ? lnp : le, 5.0f);
            lnp = le;
            has_hist = true;
        }
        h = -clampd(fabs(h) * clampd(0.9 * static_cast<double>(factor), 0.2, 5.0), 1e-8, 1e13);
    }

    unsigned long long a64 = n_att, c64 = n_acc, r64 = n_rays;
    for (int off = 16; off > 0; off >>= 1) {
        a64 += __shfl_down_sync(FULL, a64, off);
        c64 += __shfl_down_sync(FULL, c64, off);
        r64 += __shfl_down_sync(FULL, r64, off);
    }
    if (lane == 0) {
        atomicAdd(args.stats + ST_RAYS, r64);
        atomicAdd(args.stats + ST_ATTEMPTS, a64);
        atomicAdd(args.stats + ST_ACCEPTED, c64);
        atomicAdd(args.stats + ST_FP64_ATTEMPTS, a64);
    }
}

template __global__ void ms_trace_kernel<128, false, 1, 2>(MsArgs);
template __global__ void ms_trace_kernel<128, true, 1, 2>(MsArgs);
template __global__ void ms_trace_kernel<128, false, 4, 1>(MsArgs);
template __global__ void ms_trace_kernel<128, true, 4, 1>(MsArgs);
template __global__ void ms_trace_kernel<128, false, 8, 1>(MsArgs);
template __global__ void ms_trace_kernel<128, true, 8, 1>(MsArgs);

template <int G, int U>
void launch_group(MsArgs args, int sm_count, cudaStream_t s) {
    args.claim = args.claim / G > 0 ? args.claim / G : 1u;  // a warp holds 32 / G rays
    auto* kernel = args.cont.cross ? ms_trace_kernel<128, true, G, U> : ms_trace_kernel<128, false, G, U>;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 128, 0) != cudaSuccess) {
        cudaGetLastError();
        occ = 1;
    }
    kernel<<<static_cast<uint32_t>(sm_count) * static_cast<uint32_t>(occ > 1 ? occ : 1), 128, 0, s>>>(args);
}

// Lanes a ray: one, or with few rays (the launch then lasts as long as its longest
// ray's chain of attempts, each a chain of source terms) four or eight.  The lanes of
// a group repeat everything but the source terms, so this pays only while a ray has
// several sources and the groups about fit on the device at once.  FP64 at 1 / 4 / 8
// lanes (ms, means of three scenes):
//   holes    64x64             128x96            160x120           200x150           240x180
//    2    7.4 / 7.7 / 8.7   7.7 / 8.1 / 10.6  8.4 / 8.6 / 12.4  8.0 / 10.0 / 14.9 8.4 / 11.3 / 18.7
//    3    8.8 / 7.1 / 7.9   9.6 / 7.5 / 9.4   9.8 / 8.0 / 11.4  9.8 / 9.0 / 13.6  10.5 / 10.2 / 17.7
//    4   10.0 / 6.4 / 7.2  10.2 / 6.8 / 9.5  10.9 / 8.1 / 12.2 10.9 / 9.6 / 15.7  12.4 / 11.8 / 20.6
//    5   11.6 / 9.3 / 7.3  11.9 / 10.2 / 9.7 12.7 / 11.5 / 12.8 12.3 / 14.3 / 17.2 14.1 / 17.6 / 22.2
//    8   20.8 / 11.7 / 9.3 22.5 / 13.6 / 12.9 23.5 / 15.7 / 17.0 24.0 / 18.8 / 22.3 26.0 / 23.3 / 29.2
int group_lanes(uint64_t rays, uint32_t sources, int sm_count) {
    const uint64_t sm = static_cast<uint64_t>(sm_count);
    if (sources >= 5 && rays <= 32 * sm) return 8;
    if (sources >= 8 ? rays <= 192 * sm : (sources >= 3 && rays <= 160 * sm)) return 4;
    return 1;
}

}  // namespace

void launch_ms_trace(const MsArgs& args, int sm_count, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (group_lanes(args.total_rays, args.sources_per_ray, sm_count)) {
        case 8: launch_group<8, 1>(args, sm_count, s); break;
        case 4: launch_group<4, 1>(args, sm_count, s); break;
        default: launch_group<1, 2>(args, sm_count, s); break;
    }
}

}  // namespace relsim
