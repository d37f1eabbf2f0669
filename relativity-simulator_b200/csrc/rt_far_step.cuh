// rt_far_step.cuh -- the mixed tracer's far-zone Dormand-Prince attempt: FP64
// state, FP32 stages, on packed pairs of FP32 numbers.
//
// The state y and the result y5 are FP64; the stages run in FP32 on the deviation
// from free streaming:
//   x_j = x + h c_j p + h sum_m a_jm dx_m,   dx_m = (p_m - p) - 2 H s k (at stage m)
//   p_j = p + h sum_m a_jm kp_m,             kp_m = dp/dlambda (at stage m)
// so the large h p term of every position increment stays FP64 and FP32 only
// carries the gravitational part.  y5 = y + h p (FP64) + h sum b_j dx_j (FP32).
// The error estimate uses sum_j e_j = 0: E_x = h sum e_j dx_j.
//
// The far pass is bound by instruction issue and fetch, not by the FP32 pipe: an
// attempt was about 1,600 instructions around 490 FP32 operations.  sm_100's
// packed instructions (fma.rn.f32x2 and its kin) do two of them in one issue:
// components x and y of a position, momentum or null vector go in pairs, and z of
// the position with z of the momentum in the stage sums.  The reciprocals and
// roots are the bare approximations: their arguments are normal numbers in the far
// zone (r between the horizon, at least 1e-4, and 1e6), so the flushing forms give
// the same values without the rescaling of subnormals around them.
//
// Every product and sum is written with its rounding (no contraction is left to the
// compiler), so a ray's bits do not depend on how this code is scheduled or rolled.
// Measured, scalar stages / packed: 2048^2 mixed 23.9 / 21.4 ms, 1279x717 7.1 / 6.4 ms,
// a table of 40 cameras 44.4 / 39.6 ms, the 1536^2 frame with the sky 43.5 / 40.5 ms.
// One right-hand side in a loop over the stages (a third of the code) measured
// 22.5, 7.0 and 42.9 ms: its copies between stages cost more than the fetches saved.
#pragma once

#include <cuda_runtime.h>

#include "rt_device.cuh"

namespace relsim {

namespace {

__device__ __forceinline__ float f32_rsqrt(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ float f32_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) { return __ffma2_rn(pair(a), b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float a, float2 b) { return __fmul2_rn(pair(a), b); }

// A stage derivative: (dx, dy), (dkp_x, dkp_y) and (dz, dkp_z) of the deviation form.
struct FarK {
    float2 x, p, z;
};

__device__ __forceinline__ FarK far_mul(float c, const FarK& a) { return {mul2(c, a.x), mul2(c, a.p), mul2(c, a.z)}; }
__device__ __forceinline__ FarK far_fma(float c, const FarK& a, const FarK& b) {
    return {fma2(c, a.x, b.x), fma2(c, a.p, b.p), fma2(c, a.z, b.z)};
}
// c0 a + c1 b, the first product fused into the second
__device__ __forceinline__ FarK far_sum(float c0, const FarK& a, float c1, const FarK& b) {
    return far_fma(c0, a, far_mul(c1, b));
}

// Kerr-Schild right-hand side (ks_rhs) at (X, z; P, pz): the gravitational part
// -2 H s k of dx/dlambda is -th k; dp/dlambda in (dP, dpz).  Returns r.
struct FarRhs {
    float2 k, dP;
    float kz, dpz, th, hf, s;
};

__device__ __forceinline__ float far_rhs(float2 X, float z, float2 P, float pz, float M, float a, FarRhs& o) {
    const float a2 = __fmul_rn(a, a), z2 = __fmul_rn(z, z);
    float d = __fmaf_rn(X.x, X.x, __fmul_rn(X.y, X.y));
    d = __fadd_rn(__fadd_rn(d, z2), -a2);
    const float w = fmaxf(__fmaf_rn(__fmul_rn(4.0f, a2), z2, __fmul_rn(d, d)), 1e-30f);
    const float r2 = fmaxf(__fmul_rn(0.5f, __fmaf_rn(w, f32_rsqrt(w), d)), 1e-24f);
    const float inv_r = f32_rsqrt(r2);
    const float r = __fmul_rn(r2, inv_r);
    const float rpa = __fadd_rn(r2, a2);
    const float r4 = __fmul_rn(r2, r2);
    const float inv_rpa = f32_rcp(rpa);
    const float inv_den = f32_rcp(__fmaf_rn(a2, z2, r4));
    const float r3 = __fmul_rn(r2, r);
    const float H = __fmul_rn(__fmul_rn(M, r3), inv_den);
    // k = ((r x + a y), (r y - a x)) / (r^2 + a^2), z / r
    const float2 k = mul2(inv_rpa, fma2(make_float2(a, r), pair(X.y), mul2(make_float2(r, -a), pair(X.x))));
    const float kz = __fmul_rn(z, inv_r);
    const float s = __fmaf_rn(kz, pz, __fmaf_rn(k.y, P.y, __fmaf_rn(k.x, P.x, 1.0f)));
    const float th = __fmul_rn(__fmul_rn(2.0f, H), s);
    // grad r, and C, D of dH/dx_i = C dr_i (+ D for z)
    const float2 dr = mul2(__fmul_rn(r3, inv_den), X);
    const float drz = __fmul_rn(__fmul_rn(__fmul_rn(r, rpa), z), inv_den);
    const float q = __fmaf_rn(__fmul_rn(3.0f, a2), z2, -r4);
    const float C = __fmul_rn(__fmul_rn(__fmul_rn(M, r2), inv_den), __fmul_rn(q, inv_den));
    const float D = __fmul_rn(__fmul_rn(-2.0f, H), __fmul_rn(__fmul_rn(a2, z), inv_den));
    // (dk/dx_i . p) = A dr_i + B_i
    const float2 uv = fma2(-__fmul_rn(2.0f, r), k, X);
    const float wv = __fmaf_rn(uv.x, P.x, __fmul_rn(uv.y, P.y));
    const float A = __fmaf_rn(inv_rpa, wv, -__fmul_rn(__fmul_rn(inv_r, kz), pz));
    const float2 B = mul2(inv_rpa, fma2(make_float2(r, a), pair(P.x), mul2(make_float2(-a, r), pair(P.y))));
    const float Bz = __fmul_rn(inv_r, pz);
    const float s2 = __fmul_rn(s, s);
    const float G = __fmaf_rn(s2, C, __fmul_rn(th, A));
    o.dP = fma2(th, B, mul2(G, dr));
    o.dpz = __fmaf_rn(s2, D, __fmaf_rn(th, Bz, __fmul_rn(drz, G)));
    o.k = k;
    o.kz = kz;
    o.th = th;
    o.hf = H;
    o.s = s;
    return r;
}

// One stage at fraction c of the step with stage sum S: its derivative in the
// deviation form, dx = (p_j - p) - 2 H s k fused.
__device__ __forceinline__ FarK far_stage(float2 X0, float2 P0, float z0, float pz0, float h, float c, const FarK& S,
                                          float M, float a) {
    const float2 X = fma2(h, fma2(c, P0, S.x), X0);
    const float z = __fmaf_rn(h, __fmaf_rn(c, pz0, S.z.x), z0);
    const float2 dP = mul2(h, S.p);
    const float dpz = __fmul_rn(h, S.z.y);
    FarRhs f;
    far_rhs(X, z, __fadd2_rn(P0, dP), __fadd_rn(pz0, dpz), M, a, f);
    return {fma2(-f.th, f.k, dP), f.dP, make_float2(__fmaf_rn(-f.th, f.kz, dpz), f.dpz)};
}

// The attempt.  Outputs y5 and k7 in FP64 (FSAL), |E| per component, and the FP32
// BL radius, H and s of the FSAL stage at y5 (the step's bookkeeping: step cap,
// termination, projection).  A step that crosses z = 0 also gets the dense-output
// term e = h sum_j D_j k_j; sum_j D_j = 0 makes its position part h sum_j D_j dx_j,
// so it too comes from the FP32 deviations.
__device__ __forceinline__ void mixed_stages(const double* __restrict__ y, const double* __restrict__ k1, double hh,
                                             double M, double a, double* __restrict__ y5, double* __restrict__ k7,
                                             double* __restrict__ est, float& r7, float& hf7, float& s7,
                                             double* __restrict__ dense_e) {
    const float h = static_cast<float>(hh);
    const float Mf = static_cast<float>(M), af = static_cast<float>(a);
    const float2 X0 = make_float2(static_cast<float>(y[0]), static_cast<float>(y[1]));
    const float2 P0 = make_float2(static_cast<float>(y[3]), static_cast<float>(y[4]));
    const float z0 = static_cast<float>(y[2]), pz0 = static_cast<float>(y[5]);
    const FarK K1 = {make_float2(static_cast<float>(k1[0] - y[3]), static_cast<float>(k1[1] - y[4])),
                     make_float2(static_cast<float>(k1[3]), static_cast<float>(k1[4])),
                     make_float2(static_cast<float>(k1[2] - y[5]), static_cast<float>(k1[5]))};
    constexpr float C2 = 1.0f / 5.0f, C3 = 3.0f / 10.0f, C4 = 4.0f / 5.0f, C5 = 8.0f / 9.0f;
    const FarK K2 = far_stage(X0, P0, z0, pz0, h, C2, far_mul(float(DP::A21), K1), Mf, af);
    const FarK K3 = far_stage(X0, P0, z0, pz0, h, C3, far_sum(float(DP::A31), K1, float(DP::A32), K2), Mf, af);
    const FarK K4 = far_stage(X0, P0, z0, pz0, h, C4,
                              far_fma(float(DP::A43), K3, far_sum(float(DP::A41), K1, float(DP::A42), K2)), Mf, af);
    const FarK K5 = far_stage(
        X0, P0, z0, pz0, h, C5,
        far_fma(float(DP::A54), K4, far_fma(float(DP::A53), K3, far_sum(float(DP::A51), K1, float(DP::A52), K2))), Mf, af);
    const FarK K6 = far_stage(
        X0, P0, z0, pz0, h, 1.0f,
        far_fma(float(DP::A65), K5, far_fma(float(DP::A64), K4, far_fma(float(DP::A63), K3,
                far_sum(float(DP::A61), K1, float(DP::A62), K2)))), Mf, af);
    // 5th-order solution: FP64 accumulation of the FP32 increments
    const FarK Sb = far_fma(float(DP::B6), K6, far_fma(float(DP::B5), K5, far_fma(float(DP::B4), K4,
                            far_sum(float(DP::B1), K1, float(DP::B3), K3))));
    const float2 hx = mul2(h, Sb.x), hp = mul2(h, Sb.p), hz = mul2(h, Sb.z);
    const float inc[6] = {hx.x, hx.y, hz.x, hp.x, hp.y, hz.y};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        y5[i] = __dadd_rn(__fma_rn(hh, y[3 + i], y[i]), static_cast<double>(inc[i]));
        y5[3 + i] = __dadd_rn(y[3 + i], static_cast<double>(inc[3 + i]));
    }
    // stage 7 (FSAL) at y5
    FarRhs f;
    r7 = far_rhs(make_float2(static_cast<float>(y5[0]), static_cast<float>(y5[1])), static_cast<float>(y5[2]),
                 make_float2(static_cast<float>(y5[3]), static_cast<float>(y5[4])), static_cast<float>(y5[5]), Mf, af, f);
    hf7 = f.hf;
    s7 = f.s;
    const float2 gk = mul2(-f.th, f.k);
    const float g[6] = {gk.x, gk.y, __fmul_rn(-f.th, f.kz), f.dP.x, f.dP.y, f.dpz};
    FarK K7;
    K7.x = make_float2(__fadd_rn(static_cast<float>(__dsub_rn(y5[3], y[3])), g[0]),
                       __fadd_rn(static_cast<float>(__dsub_rn(y5[4], y[4])), g[1]));
    K7.p = f.dP;
    K7.z = make_float2(__fadd_rn(static_cast<float>(__dsub_rn(y5[5], y[5])), g[2]), f.dpz);
    const FarK Se = far_fma(float(DP::E7), K7, far_fma(float(DP::E6), K6, far_fma(float(DP::E5), K5,
                            far_fma(float(DP::E4), K4, far_sum(float(DP::E1), K1, float(DP::E3), K3)))));
    const float2 ex = mul2(h, Se.x), ep = mul2(h, Se.p), ez = mul2(h, Se.z);
    const float e[6] = {ex.x, ex.y, ez.x, ep.x, ep.y, ez.y};
#pragma unroll
    for (int i = 0; i < 6; ++i) est[i] = static_cast<double>(fabsf(e[i]));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        k7[i] = __dadd_rn(y5[3 + i], static_cast<double>(g[i]));
        k7[3 + i] = static_cast<double>(g[3 + i]);
    }
    if (y[2] * y5[2] <= 0.0) {
        const FarK Sd = far_fma(float(DP::D7), K7, far_fma(float(DP::D6), K6, far_fma(float(DP::D5), K5,
                                far_fma(float(DP::D4), K4, far_sum(float(DP::D3), K3, float(DP::D1), K1)))));
        const float2 dx = mul2(h, Sd.x), dp = mul2(h, Sd.p), dz = mul2(h, Sd.z);
        dense_e[0] = static_cast<double>(dx.x);
        dense_e[1] = static_cast<double>(dx.y);
        dense_e[2] = static_cast<double>(dz.x);
        dense_e[3] = static_cast<double>(dp.x);
        dense_e[4] = static_cast<double>(dp.y);
        dense_e[5] = static_cast<double>(dz.y);
    }
}

}  // namespace

}  // namespace relsim
