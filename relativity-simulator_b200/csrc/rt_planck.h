// rt_planck.h -- the blackbody colour of the disk and the torus: Planck radiance
// against the 33-node spectral table (accretion_disk_model.hpp:71-88), host/device,
// and a table of it for the device.
//
// A colour is 33 exponentials and 66 divisions, about 2,000 FP64 instructions, and
// depends on the temperature alone (the nodes and weights are constants).  The
// torus asks for one at every sample of every chord.  With s = 1 / T, s * xyz(s) is
// smooth and locally exponential: on pieces of s of width 2^-17 / K, up to 1 / 500 K,
// degree-8 interpolants at Chebyshev nodes reproduce it (remainder 2 (de / 4)^9 / 9!,
// below 4e-16 for the bluest node's exponent change de = 0.29 over a piece).  27 fused
// operations and one reciprocal replace the sum.
//
// The table is the more accurate of the two.  Its values are formed in extended
// precision; a piece's width is a power of two, so that the place within a piece is
// exact, and the rounding of 1 / T, which the exponents of up to 76 multiply, is taken
// back out.  Largest and mean relative error over 500 to 400,000 K: the sum 5.3e-15 and
// 2.5e-16, the table 3.3e-16 and 6.5e-17.  Colder than 500 K, where the sum drops nodes, it
// is evaluated as it stands.
// Measured with the closed forms of the torus's fluid (rt_torus.cuh), a 640x360 frame:
// 68.1 ms before, 35.5 after.
#pragma once

#include <cmath>
#include <cstdint>

#include "rt_fast_math.h"

#ifdef __CUDACC__
#define RT_PL_HD __host__ __device__
#else
#define RT_PL_HD
#endif

namespace relsim {

constexpr double kPlanckC2 = 14387.76877;  // second radiation constant, um K

// Planck sum against the spectral table (wavelengths in um, weights per node): XYZ.
RT_PL_HD inline void planck_sum(const double* lambda_um, const double (*w)[3], double temperature_k, double* xyz) {
    const double t = temperature_k < 300.0 ? 300.0 : (400000.0 < temperature_k ? 400000.0 : temperature_k);
    xyz[0] = xyz[1] = xyz[2] = 0.0;
    for (int i = 0; i <= 32; ++i) {
        const double lum = lambda_um[i];
        const double e = kPlanckC2 / (lum * t);
        if (e > 80.0) continue;
        const double l2 = lum * lum;
        const double rad = 1.0 / (l2 * l2 * lum * expm1(e));
        xyz[0] += rad * w[i][0];
        xyz[1] += rad * w[i][1];
        xyz[2] += rad * w[i][2];
    }
}

constexpr int kPlanckPieces = 263, kPlanckTerms = 9, kPlanckStride = 28;  // doubles a piece, 16-byte aligned
constexpr int kPlanckTableDoubles = kPlanckPieces * kPlanckStride;
constexpr double kPlanckMinT = 500.0;
constexpr double kPlanckPerS = 131072.0;  // pieces per unit of s
static_assert(kPlanckPerS / kPlanckMinT < kPlanckPieces, "pieces up to 1 / kPlanckMinT");

// Fill the table: per piece, the power-basis coefficients (lowest first, x y z
// together) of s * xyz in u = 2 * (place within the piece) - 1.
inline void planck_table_fill(const double* lambda_um, const double (*w)[3], double* table) {
    using Real = long double;
    constexpr int N = kPlanckTerms;
    const Real pi = 3.14159265358979323846264338327950288L;
    Real node[N], cosine[N][N], power[N][N] = {};  // power[k]: T_k in powers of u
    for (int j = 0; j < N; ++j) node[j] = std::cos(pi * (j + Real(0.5)) / N);
    for (int k = 0; k < N; ++k)
        for (int j = 0; j < N; ++j) cosine[k][j] = std::cos(pi * k * (j + Real(0.5)) / N);
    power[0][0] = power[1][1] = 1;
    for (int k = 2; k < N; ++k)
        for (int m = 0; m < N; ++m) power[k][m] = (m > 0 ? 2 * power[k - 1][m - 1] : Real(0)) - power[k - 2][m];
    // e^x at the first piece's places and its factor from piece to piece, per node
    Real grow[33], ex[N][33];
    for (int i = 0; i <= 32; ++i) {
        grow[i] = std::exp(kPlanckC2 / (Real(lambda_um[i]) * kPlanckPerS));
        for (int j = 0; j < N; ++j)
            ex[j][i] = std::exp(kPlanckC2 * (Real(0.5) + Real(0.5) * node[j]) / (Real(lambda_um[i]) * kPlanckPerS));
    }
    for (int p = 0; p < kPlanckPieces; ++p) {
        Real value[N][3] = {};
        for (int j = 0; j < N; ++j) {
            const Real s = (p + Real(0.5) + Real(0.5) * node[j]) / kPlanckPerS;
            for (int i = 0; i <= 32; ++i) {
                const Real lum = lambda_um[i], l2 = lum * lum;
                const Real rad = s / (l2 * l2 * lum * (ex[j][i] - 1));
                ex[j][i] *= grow[i];
                for (int c = 0; c < 3; ++c) value[j][c] += rad * w[i][c];
            }
        }
        double* out = table + p * kPlanckStride;
        for (int i = 0; i < kPlanckStride; ++i) out[i] = 0.0;
        for (int c = 0; c < 3; ++c) {
            Real coeff[N] = {};
            for (int k = 0; k < N; ++k) {
                Real a = 0;
                for (int j = 0; j < N; ++j) a += value[j][c] * cosine[k][j];
                a *= Real(k == 0 ? 1 : 2) / N;
                for (int m = 0; m < N; ++m) coeff[m] += a * power[k][m];
            }
            for (int m = 0; m < N; ++m) out[3 * m + c] = static_cast<double>(coeff[m]);
        }
    }
}

// XYZ from the table for kPlanckMinT <= t (clamped to 400,000 K above).
RT_PL_HD inline void planck_lookup(const double* __restrict__ table, double temperature_k, double* xyz) {
    const double t = 400000.0 < temperature_k ? 400000.0 : temperature_k;
    const double s = fast_rcp(t);
    const double at = s * kPlanckPerS;  // exact, and so is the place within the piece
    int p = static_cast<int>(at);
    p = p < 0 ? 0 : (p > kPlanckPieces - 1 ? kPlanckPieces - 1 : p);
    const double place = 2.0 * (at - static_cast<double>(p)) - 1.0;
    const double u = fma(2.0 * at, fma(-t, s, 1.0), place);  // 1 / t is s + s (1 - t s)
    const double* __restrict__ c = table + p * kPlanckStride;
    double v[kPlanckStride];
#ifdef __CUDA_ARCH__
    const double2* __restrict__ c2 = reinterpret_cast<const double2*>(c);
#pragma unroll
    for (int i = 0; i < kPlanckStride / 2; ++i) {
        const double2 q = __ldg(c2 + i);
        v[2 * i] = q.x;
        v[2 * i + 1] = q.y;
    }
#else
    for (int i = 0; i < kPlanckStride; ++i) v[i] = c[i];
#endif
    for (int k = 0; k < 3; ++k) {
        double q = v[3 * (kPlanckTerms - 1) + k];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int m = kPlanckTerms - 2; m >= 0; --m) q = fma(q, u, v[3 * m + k]);
        xyz[k] = q * t;
    }
}

}  // namespace relsim
