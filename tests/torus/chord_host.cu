// One chord's light through the torus (fm_chord, rt_shade.cuh) on the host and on the
// device, beside the chord integral as the reference writes it (hydro_disk_shading.hpp:173-269,
// hydro/fishbone_moncrief.hpp:118-224, accretion_disk_model.hpp:71-88 and :218-221),
// here in double and in extended precision.  Test-only.
#include <cmath>
#include <vector>

#include "rt_shade.cuh"

using namespace relsim;

namespace chord_test {

template <class R>
R within(R v, R lo, R hi) {
    return v < lo ? lo : (hi < v ? hi : v);
}

// Light of one chord: radiance r, g, b, opacity and the weighted redshift; false: none.
template <class R>
bool chord(const ShadeDesc& D, const double* from, const double* to, double l_over_e, R out[5]) {
    const R f[3] = {from[0], from[1], from[2]};
    const R d[3] = {to[0] - f[0], to[1] - f[1], to[2] - f[2]};
    const R len2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    if (len2 < R(1e-24)) return false;
    const R len = std::sqrt(len2), outer = D.fm_outer, m = D.fm_m, a = D.fm_a, l = D.fm_l;
    const R b = (f[0] * d[0] + f[1] * d[1] + f[2] * d[2]) / len2;
    const R c = (f[0] * f[0] + f[1] * f[1] + f[2] * f[2] - outer * outer) / len2;
    const R disc = b * b - c;
    if (disc <= 0) return false;
    const R root = std::sqrt(disc);
    const R t0 = within<R>(-b - root, 0, 1), t1 = within<R>(-b + root, 0, 1);
    if (t1 <= t0) return false;
    const R clipped = len * (t1 - t0);
    int count = static_cast<int>(std::ceil(clipped * D.fm_density / m));
    count = count < 1 ? 1 : (count > 128 ? 128 : count);
    const R step = clipped / count;
    const float* P = D.profile;
    const R span = std::max<R>(D.fm_h_max - R(1), R(1e-12));
    R rad[3] = {0, 0, 0}, trans = 1, wsum = 0, zsum = 0;
    for (int i = 0; i < count; ++i) {
        const R t = t0 + (t1 - t0) * ((i + R(0.5)) / count);
        const R x = f[0] + t * d[0], y = f[1] + t * d[1], z = f[2] + t * d[2];
        const R r = std::sqrt(x * x + y * y + z * z);
        if (r < D.fm_inner || r > outer) continue;
        const R theta = std::acos(within<R>(z / r, -1, 1));
        const R st = std::sin(theta), ct = std::cos(theta), s2 = std::max<R>(st * st, R(1e-30)), c2 = ct * ct;
        const R r2 = r * r, a2 = a * a, rho2 = r2 + a2 * c2, delta = r2 - 2 * m * r + a2;
        const R sigma = (r2 + a2) * (r2 + a2) - a2 * delta * s2;
        const R den = sigma * s2 - 4 * m * r * a * l * s2 - l * l * (delta - a2 * s2);
        if (r <= R(D.fm_rh) * R(1.0001) || den <= 0 || delta <= 0) continue;
        const R w = R(0.5) * std::log(std::max<R>((rho2 * delta * s2) / den, R(1e-30)));
        if (w >= D.fm_w_in) continue;
        const R h = std::exp(D.fm_w_in - w);
        if (!(h > R(1) + R(1e-9))) continue;
        const R ratio = within<R>((h - 1) / span, 0, 1);
        const R tau = D.fm_kappa * std::pow(ratio, R(D.fm_exponent)) * step / m;
        if (tau < R(1e-12)) continue;
        const R lt = -std::exp(w), lphi = -l * lt;
        const R gtt = -sigma / (rho2 * delta), gtp = -(2 * m * r * a) / (rho2 * delta);
        const R gpp = (delta - a2 * s2) / (rho2 * delta * s2);
        const R ut = gtt * lt + gtp * lphi, uphi = gtp * lt + gpp * lphi;
        if (ut <= R(1e-12)) continue;
        const R q = ut * (1 - (uphi / ut) * l_over_e);
        const R g = (std::fabs(q) > R(1e-9)) ? within<R>(1 / q, R(0.05), 4) : R(1);
        const R kelvin = (R(P[DP_FLOOR_T]) + (R(P[DP_PEAK_T]) - R(P[DP_FLOOR_T])) * ratio) * g;
        R xyz[3] = {0, 0, 0};
        for (int k = 0; k <= 32; ++k) {
            const R lum = D.lambda_um[k], l2 = lum * lum, e = R(kPlanckC2) / (lum * within<R>(kelvin, 300, 400000));
            if (e > 80) continue;
            const R radiance = 1 / (l2 * l2 * lum * std::expm1(e));
            for (int j = 0; j < 3; ++j) xyz[j] += radiance * D.weight[k][j];
        }
        const R inv = 1 / std::max<R>(R(P[DP_REF_LUMINANCE]), R(1e-30));
        const R gain = R(P[DP_BRIGHTNESS]) * std::pow(g, R(P[DP_BEAMING]));
        const R X = xyz[0] * inv, Y = xyz[1] * inv, Z = xyz[2] * inv;
        R col[3] = {std::max<R>(R(3.2404542) * X - R(1.5371385) * Y - R(0.4985314) * Z, 0) * gain,
                    std::max<R>(R(-0.9692660) * X + R(1.8760108) * Y + R(0.0415560) * Z, 0) * gain,
                    std::max<R>(R(0.0556434) * X - R(0.2040259) * Y + R(1.0572252) * Z, 0) * gain};
        const R luma = R(0.2126) * col[0] + R(0.7152) * col[1] + R(0.0722) * col[2];
        const R through = std::exp(-tau), weight = trans * (1 - through);
        for (int j = 0; j < 3; ++j) {
            const R graded = std::max<R>(0, luma + (col[j] - luma) * R(P[DP_SATURATION]));
            rad[j] += weight * graded * (1 + (R(P[DP_TINT_R + j]) - 1) * R(P[DP_TINT_STRENGTH]));
        }
        wsum += weight;
        zsum += weight * g;
        trans *= through;
        if (trans < R(0.002)) break;
    }
    if (1 - trans <= R(1e-6)) return false;
    for (int j = 0; j < 3; ++j) out[j] = rad[j];
    out[3] = 1 - trans;
    out[4] = wsum > R(1e-30) ? zsum / wsum : R(1);
    return true;
}

// The descriptor of a unit hole's torus; the table is the caller's.
ShadeDesc descriptor(double spin, double gamma, const double* lambda_um, const double* weight, const float* disk) {
    ShadeDesc D{};
    const torus::TorusContext c = torus::make_torus(1.0, spin, 6.0, 12.0);
    for (int i = 0; i < 33; ++i) {
        D.lambda_um[i] = lambda_um[i];
        for (int j = 0; j < 3; ++j) D.weight[i][j] = weight[3 * i + j];
    }
    for (int i = 0; i < 32; ++i) D.profile[i] = disk[i];
    D.mass = 1.0;
    D.disk_spin = spin;
    set_torus(D, c, gamma, 0.35, 2.0);
    return D;
}

struct Light {
    double v[5], any;
};

__host__ __device__ Light light_of(const ShadeDesc& D, const double* v) {
    ChordLight c{};
    const bool any = fm_chord(D, v, v + 3, v[6], c);
    return {{c.rad[0], c.rad[1], c.rad[2], c.opacity, c.z}, any ? 1.0 : 0.0};
}

__global__ void chord_kernel(const ShadeDesc* D, const double* chords, long n, Light* out) {
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if (i < n) out[i] = light_of(*D, chords + 7 * i);
}

bool on_device(ShadeDesc D, const double* table, const double* chords, long n, Light* out) {
    char* mem = nullptr;
    const size_t t = sizeof(double) * kPlanckTableDoubles, d = sizeof(ShadeDesc), c = sizeof(double) * 7 * n;
    if (cudaMalloc(&mem, t + d + c + sizeof(Light) * n) != cudaSuccess) return false;
    D.planck = reinterpret_cast<double*>(mem);
    cudaMemcpy(mem, table, t, cudaMemcpyHostToDevice);
    cudaMemcpy(mem + t, &D, d, cudaMemcpyHostToDevice);
    cudaMemcpy(mem + t + d, chords, c, cudaMemcpyHostToDevice);
    chord_kernel<<<static_cast<unsigned>((n + 63) / 64), 64>>>(reinterpret_cast<ShadeDesc*>(mem + t),
                                                             reinterpret_cast<double*>(mem + t + d), n,
                                                             reinterpret_cast<Light*>(mem + t + d + c));
    const cudaError_t e = cudaMemcpy(out, mem + t + d + c, sizeof(Light) * n, cudaMemcpyDeviceToHost);
    cudaFree(mem);
    return e == cudaSuccess;
}

}  // namespace chord_test

using namespace chord_test;

// n chords (from and to, l_over_e) through the torus of a unit hole, fm_chord on the host or
// the device; lambda_um, weight and disk are the spectral table and the disk profile.  err:
// [2][5][n], the errors of the light (in parts of an opaque chord's), of the opacity and of
// the redshift against extended precision: fm_chord's, then those of the same integral in
// double; -1 where no light.  Returns the chords on which the three do not agree whether
// there is any; negative: the device did not run.
extern "C" long chords(int device, double spin, double gamma, const double* lambda_um, const double* weight,
                       const float* disk, long n, const double* ends, double* err) {
    static double table[kPlanckTableDoubles];
    ShadeDesc D = descriptor(spin, gamma, lambda_um, weight, disk);
    planck_table_fill(D.lambda_um, D.weight, table);
    std::vector<Light> ours(n);
    if (device) {
        if (!on_device(D, table, ends, n, ours.data())) return -1;
    } else {
        D.planck = table;
        for (long i = 0; i < n; ++i) ours[i] = light_of(D, ends + 7 * i);
    }
    long odd = 0;
    for (long i = 0; i < n; ++i) {
        const double* v = ends + 7 * i;
        double plain[5];
        long double exact[5];
        const bool a = ours[i].any != 0.0;
        const bool b = chord<double>(D, v, v + 3, v[6], plain), e = chord<long double>(D, v, v + 3, v[6], exact);
        odd += a != e || b != e;
        for (int k = 0; k < 5; ++k) {
            const long double whole = k < 3 ? exact[k] / exact[3] : 1.0L;
            const bool has = a && b && e && whole > 0;
            err[k * n + i] = has ? static_cast<double>(fabsl(ours[i].v[k] - exact[k]) / whole) : -1.0;
            err[(5 + k) * n + i] = has ? static_cast<double>(fabsl(plain[k] - exact[k]) / whole) : -1.0;
        }
    }
    return odd;
}
