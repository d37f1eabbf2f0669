// rt_trace.cu -- persistent backward null-geodesic tracer for sm_100a.
//
// One ray per lane.  Warps claim rays from a global work counter; when at
// least `refill_threshold` lanes of a warp are idle the warp claims that many
// consecutive rays with one atomic (ballot + popc rank), so lanes whose rays
// terminated are refilled instead of idling while the warp's longest ray runs.
//
// Per ray: Dormand-Prince 5(4) on the Kerr-Schild Hamiltonian state (x, p)
// with p_t = -1 (kerr_schild_null_integrator.hpp:72-114), PI30 control
// (step_controller.hpp:51-58; accept/reject scaling rk45_adaptive.hpp:294-310),
// FSAL reuse of the last stage, a step cap |h| <= c max(r - r_+, 0.01 M),
// projection onto H = 0 after each accepted step, and classification:
// captured (r < capture_scale r_+, software_compute_engine.hpp:1667-1671),
// escaped (r > escape radius, :1672-1675), disk (first z = 0 crossing on
// [r_in, r_out], root by Illinois regula falsi on the DP5 solution of a step
// fraction), with the Carter certain-capture early-out
// (carter_ray_classifier.hpp:146-150).  Terminal points are interpolated to
// the threshold radius (cubic Hermite on the step's FSAL end points).
//
// Layout: the hot state (y, k1, r, h, counters) lives in registers; cold
// per-lane state (affine parameter, invariants at the start, root bracket) in
// shared memory as structure of arrays.  Ray set-up, termination and the
// Carter test are out of line so the step loop stays small in the
// instruction cache; states cross that boundary through small local arrays.
// The disk root solve reuses the loop's stage code: a lane in ROOT mode runs
// its next DP5 evaluation at a fraction of the step instead of a full step.
//
// The mixed-precision mode runs as two passes (PASS_FAR, PASS_NEAR) instead:
// an FP32-stage kernel for the far zone and an FP64 kernel for the zone near
// the hole, rays moving between them through queues with their state parked
// in HBM, disk crossings solved on the step's dense output, and disk hits
// written by a finish kernel.  Splitting the code this way keeps each loop
// small in the instruction cache (the single mixed kernel, which holds both
// step forms, is instruction-fetch bound).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "rt_device.cuh"
#include "rt_far_step.cuh"
#include "rt_internal.h"
#include "rt_ray.cuh"

namespace relsim {

namespace {

// Dormand-Prince tableau rows for the rolled FP64 step: row s gives the
// coefficients of k1..k(s+1) in the input of stage s + 2 (row 5 = b, the
// 5th-order solution); kDpE are the error weights of k1..k7.
__constant__ double kDpA[6][6] = {
    {DP::A21, 0, 0, 0, 0, 0},
    {DP::A31, DP::A32, 0, 0, 0, 0},
    {DP::A41, DP::A42, DP::A43, 0, 0, 0},
    {DP::A51, DP::A52, DP::A53, DP::A54, 0, 0},
    {DP::A61, DP::A62, DP::A63, DP::A64, DP::A65, 0},
    {DP::B1, 0.0, DP::B3, DP::B4, DP::B5, DP::B6}};
__constant__ double kDpE[7] = {DP::E1, 0.0, DP::E3, DP::E4, DP::E5, DP::E6, DP::E7};

// Stage derivatives k2..k7 of the rolled FP64 step, per thread in shared memory.
template <int BLOCK>
struct KStore {
    double k[6][6][BLOCK];
};

// FP64 stages 2..7 as one rolled loop around a single RHS (small in the
// instruction cache; used where FP64 steps are a minority, e.g. the near zone
// of the mixed mode).  Same arithmetic as the straight-line form.
template <int BLOCK>
__device__ __forceinline__ void fp64_stages_rolled(const double* __restrict__ y, const double* __restrict__ k1,
                                                   double hh, double M, double a, KStore<BLOCK>& K, int tid,
                                                   bool root, double* __restrict__ y5, double* __restrict__ k7,
                                                   double* __restrict__ est, double& r5, double& hf5, double& s5) {
#pragma unroll 1
    for (int st = 0; st < 6; ++st) {
        double in[6];
        // the stage sum unrolled over j (predicated on j <= st): the shared-memory loads
        // of a stage are independent and issue up front instead of one per FMA
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double acc = kDpA[st][0] * k1[i];
#pragma unroll
            for (int j = 1; j < 6; ++j)
                if (j <= st) acc += kDpA[st][j] * K.k[j - 1][i][tid];
            in[i] = y[i] + hh * acc;
        }
        if (st == 5) {
#pragma unroll
            for (int i = 0; i < 6; ++i) y5[i] = in[i];
            if (root) return;
        }
        double out[6], hf, sv;
        const double rr = ks_rhs(in, M, a, out, hf, sv);
#pragma unroll
        for (int i = 0; i < 6; ++i) K.k[st][i][tid] = out[i];
        if (st == 5) {
#pragma unroll
            for (int i = 0; i < 6; ++i) k7[i] = out[i];
            r5 = rr;
            hf5 = hf;
            s5 = sv;
        }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        double acc = kDpE[0] * k1[i];
#pragma unroll
        for (int j = 2; j < 7; ++j) acc += kDpE[j] * K.k[j - 1][i][tid];
        est[i] = fabs(hh) * fabs(acc);
    }
}

// FP64 stages 2..7, straight-line (rk45_adaptive.hpp:210-252).  A root evaluation
// stops at y5.  DENSE: a step that crosses z = 0 also gets its dense-output term.
template <bool FAST, bool DENSE>
__device__ __forceinline__ void fp64_stages(const double* __restrict__ y, const double* __restrict__ k1, double hh,
                                            double M, double a, bool root, double* __restrict__ y5,
                                            double* __restrict__ kA, double* __restrict__ est,
                                            double* __restrict__ dense5, double& r5, double& hf5, double& s5) {
    double k3[6], k4[6], k5[6], k6[6];
    double in[6], hf, sv;
#pragma unroll
    for (int i = 0; i < 6; ++i) in[i] = y[i] + hh * (DP::A21 * k1[i]);
    ks_rhs<FAST>(in, M, a, kA, hf, sv);
#pragma unroll
    for (int i = 0; i < 6; ++i) in[i] = y[i] + hh * (DP::A31 * k1[i] + DP::A32 * kA[i]);
    ks_rhs<FAST>(in, M, a, k3, hf, sv);
#pragma unroll
    for (int i = 0; i < 6; ++i) in[i] = y[i] + hh * (DP::A41 * k1[i] + DP::A42 * kA[i] + DP::A43 * k3[i]);
    ks_rhs<FAST>(in, M, a, k4, hf, sv);
#pragma unroll
    for (int i = 0; i < 6; ++i)
        in[i] = y[i] + hh * (DP::A51 * k1[i] + DP::A52 * kA[i] + DP::A53 * k3[i] + DP::A54 * k4[i]);
    ks_rhs<FAST>(in, M, a, k5, hf, sv);
#pragma unroll
    for (int i = 0; i < 6; ++i)
        in[i] = y[i] + hh * (DP::A61 * k1[i] + DP::A62 * kA[i] + DP::A63 * k3[i] + DP::A64 * k4[i] + DP::A65 * k5[i]);
    ks_rhs<FAST>(in, M, a, k6, hf, sv);
#pragma unroll
    for (int i = 0; i < 6; ++i)
        y5[i] = y[i] + hh * (DP::B1 * k1[i] + DP::B3 * k3[i] + DP::B4 * k4[i] + DP::B5 * k5[i] + DP::B6 * k6[i]);
    if (!root) {
        r5 = ks_rhs<FAST>(y5, M, a, kA, hf5, s5);
#pragma unroll
        for (int i = 0; i < 6; ++i)
            est[i] = fabs(hh) * fabs(DP::E1 * k1[i] + DP::E3 * k3[i] + DP::E4 * k4[i] + DP::E5 * k5[i] +
                                     DP::E6 * k6[i] + DP::E7 * kA[i]);
        if constexpr (DENSE) {
            if (y[2] * y5[2] <= 0.0) {
#pragma unroll
                for (int i = 0; i < 6; ++i)
                    dense5[i] = hh * (DP::D1 * k1[i] + DP::D3 * k3[i] + DP::D4 * k4[i] + DP::D5 * k5[i] +
                                      DP::D6 * k6[i] + DP::D7 * kA[i]);
            }
        }
    }
}

// The same attempt with the compiler's division and square root, for an attempt whose
// stages leave the fast forms' range: out of line, y and k1 in io[0..11], then y5, k7,
// est, the dense-output term, r, H and s.
template <bool DENSE>
__device__ __noinline__ void fp64_stages_special(double* __restrict__ io, double hh, double M, double a, bool root) {
    double y[6], k1[6], y5[6], kA[6], est[6], dense5[6], r5 = 0.0, hf5 = 0.0, s5 = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        y[i] = io[i];
        k1[i] = io[6 + i];
        kA[i] = est[i] = dense5[i] = 0.0;
    }
    fp64_stages<false, DENSE>(y, k1, hh, M, a, root, y5, kA, est, dense5, r5, hf5, s5);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        io[12 + i] = y5[i];
        io[18 + i] = kA[i];
        io[24 + i] = est[i];
        io[30 + i] = dense5[i];
    }
    io[36] = r5;
    io[37] = hf5;
    io[38] = s5;
}

}  // namespace

// Store the end of a ray's accepted step (after a gap its start too) in its chain of
// pages (PathOut); the page is S.side, the count S.rit (both idle: a torus-shaded trace
// has no disk roots).  False: no free page; the ray is in the overflow queue and its
// steps are off the counters.
constexpr int kPathGap = 1 << 30;  // in S.rit: steps were left out since the last point
template <class ColdT>
__device__ __noinline__ bool store_path_points(const TraceArgs& args, ColdT& S, int tid, uint64_t ray,
                                               uint32_t acc, uint32_t rej, const double* x) {
    const PathOut& P = args.path;
    const uint64_t local = S.local[tid];
    uint32_t k = static_cast<uint32_t>(S.rit[tid] & ~kPathGap);
    double* page = P.pages + static_cast<uint64_t>(S.side[tid]) * kPathPageDoubles;
    for (int i = (S.rit[tid] & kPathGap) ? 0 : 2; i < 3; ++i, ++k) {  // gap, start, end
        const uint32_t slot = k % kPathPoints;
        if (slot == 0) {
            const uint32_t next = atomicAdd(P.cursor + PC_PAGE, 1u);
            if (next >= P.capacity) {
                P.overflow[atomicAdd(P.cursor + PC_OVERFLOW, 1u)] = static_cast<uint32_t>(ray);
                const unsigned long long att = static_cast<unsigned long long>(acc) + rej;
                atomicAdd(args.stats + ST_ATTEMPTS, 0ull - att);
                atomicAdd(args.stats + ST_FP64_ATTEMPTS, 0ull - att);
                atomicAdd(args.stats + ST_ACCEPTED, 0ull - acc);
                atomicAdd(args.stats + ST_RHS, 0ull - (6 * att + 1));
                return false;
            }
            if (k == 0) P.first[local] = next;
            else page[3 * kPathPoints] = static_cast<double>(next);
            S.side[tid] = static_cast<int>(next);
            page = P.pages + static_cast<uint64_t>(next) * kPathPageDoubles;
        }
        double* at = page + 3 * slot;
        at[0] = (i == 0) ? __longlong_as_double(0x7ff8000000000000ll) : x[3 * (i - 1)];
        at[1] = x[i == 0 ? 1 : 3 * (i - 1) + 1];
        at[2] = x[i == 0 ? 2 : 3 * (i - 1) + 2];
    }
    S.rit[tid] = static_cast<int>(k);
    return true;
}

// The light of four rays of a torus-shaded trace by one warp (local: this lane's ray,
// the same in the eight lanes of its group; points 0: none).  A group walks its ray's
// chain eight points at a time, one chord to a lane (fm_chord), and adds the chords'
// light in the order of the steps.  Gathering inside the step loop ran two large pieces
// of code in turn on every warp, each evicting the other from the instruction cache
// (no_instruction 3.5 of 9.6 cycles per issue, FP64 pipe 26 %); one lane to a ray left
// the pass to the few rays along the equatorial plane (4.5 ms at 640x360, the SMs idle
// for two thirds of it).  Measured, gathering as it goes / a pass after the trace, one
// lane to a ray / eight lanes, idle warps of the trace first: 64x36 14.6 / 10.1 / 3.0 ms,
// 640x360 32.7 / 17.3 / 13.6, 1920x1080 159 / 76 / 67.  Sixteen lanes: the same, 77.
constexpr int kPathLanes = 8;
__device__ __forceinline__ void sample_paths(const TraceArgs& args, uint32_t local, uint32_t points) {
    constexpr unsigned FULL = 0xffffffffu;
    const BundleDesc& B = args.one;
    const int sub = threadIdx.x % kPathLanes;
    const uint64_t o = B.out_offset + local;
    double x[3], last[3], V[VL_COUNT] = {}, lz = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) x[c] = B.x0[c];
    bl_cartesian(x, B.a, last);  // the end of the group's last chord
    const double* page = args.path.pages;
    if (points) {
        lz = args.cont.lz[o];
        page += static_cast<uint64_t>(args.path.first[local]) * kPathPageDoubles;
    }
    bool open = points != 0;
    for (uint32_t k = 0; __any_sync(FULL, open); k += kPathLanes) {
        const uint32_t slot = k % kPathPoints;
        double to[3], from[3];
        bool live = open && k + sub < points;
        if (open && slot == 0 && k)
            page = args.path.pages + static_cast<uint64_t>(page[3 * kPathPoints]) * kPathPageDoubles;
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = live ? page[3 * (slot + sub) + c] : 1.0;
        bl_cartesian(x, B.a, to);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double before = __shfl_up_sync(FULL, to[c], 1, kPathLanes);
            from[c] = sub ? before : last[c];
            last[c] = __shfl_sync(FULL, to[c], kPathLanes - 1, kPathLanes);
        }
        live = live && to[0] == to[0] && from[0] == from[0];  // not beside a gap
        ChordLight light;
        const bool lit = live && fm_chord(*args.cont.shade, from, to, lz, light);
        const unsigned any = __ballot_sync(FULL, lit);
        unsigned mine = (any >> (threadIdx.x % 32 - sub)) & ((1u << kPathLanes) - 1u);
        while (__any_sync(FULL, mine != 0u)) {
            const int j = mine ? __ffs(mine) - 1 : 0;
            ChordLight c;
#pragma unroll
            for (int f = 0; f < 3; ++f) c.rad[f] = __shfl_sync(FULL, light.rad[f], j, kPathLanes);
            c.opacity = __shfl_sync(FULL, light.opacity, j, kPathLanes);
            c.z = __shfl_sync(FULL, light.z, j, kPathLanes);
            if (mine && open) {
                fm_add(c, V);
                open = fm_open(V);
            }
            mine &= mine - 1u;
        }
        open = open && k + kPathLanes < points;
    }
    if (points && sub < VL_COUNT) {
        double v = V[0];
#pragma unroll
        for (int f = 1; f < VL_COUNT; ++f) v = (sub == f) ? V[f] : v;
        args.cont.vol[o * VL_COUNT + sub] = v;
    }
}

// A warp of a torus-shaded trace that finds no more rays: while others still trace, it
// samples the rays that have ended, four of the launch's order at a time.  Nothing is
// waited for: a ray that has not ended when its turn comes is left to the sampling pass,
// and so is all the rest once the last warp's rays have ended.
__device__ __noinline__ void sample_ended_paths(const TraceArgs& args) {
    const PathOut& P = args.path;
    const int lane = threadIdx.x & 31;
    const uint32_t total = static_cast<uint32_t>(args.total_rays), warps = gridDim.x * (blockDim.x / 32u);
    if (lane == 0) atomicAdd(P.cursor + PC_IDLE_WARPS, 1u);
    for (;;) {
        uint32_t at = total;
        if (lane == 0 && *static_cast<volatile uint32_t*>(P.cursor + PC_IDLE_WARPS) < warps)
            at = atomicAdd(P.cursor + PC_SAMPLED, 32u / kPathLanes);
        at = __shfl_sync(~0u, at, 0);
        if (at >= total) return;
        const uint32_t i = at + lane / kPathLanes;
        uint32_t local = 0, points = 0;
        if (i < total) {
            local = P.order[i];
            if (lane % kPathLanes == 0) points = *static_cast<volatile uint32_t*>(P.points + local);
        }
        points = __shfl_sync(~0u, points, 0, kPathLanes);
        if (points == kPathOpen) points = 0;
        __threadfence();  // the chain was stored before its length
        __syncwarp();     // and the group's other lanes read it after the one that saw that
        sample_paths(args, local, points);
        if (points && lane % kPathLanes == 0) P.points[local] = 0;  // gathered
        __syncwarp();
    }
}

// WARPS resident warps per SM set the registers per thread: 8 warps at up to 255
// registers, 12 at 168, 16 at 128.  Fewer warps spill less and an attempt takes less
// time; more warps hide more of the FP64 latency that bounds the step loop.
//
//   12: the general case; it spills a little.
//   16: the plain FP64 tracer over many rays (kWideRaysPerSm).  In the far, near and
//       critical passes it loses (1279x717: 4.53 / 4.71, 0.89 / 1.19 and 1.73 / 2.01
//       ms at 12 / 16): their warps run few rays or few lanes.
//    8: launches of few rays, which last as long as their longest ray
//       (kLeanRaysPerSm, kLeanMixedRaysPerSm).
//
// PASS selects the single-kernel tracer or one pass of the two-pass mixed
// tracer.  The far pass (FP32 stages only) parks a ray when it enters the FP64
// zone; the near pass (FP64 stages) parks it back when it leaves the zone
// again.  Both passes solve disk crossings on the step's dense output.  Parked
// rays resume from their saved state, so a ray's arithmetic does not depend on
// which rays share its warp.
//
// ONE: a launch of one camera, its descriptor among the kernel's parameters: the step
// loop's dozen constants are operands from the constant bank instead of loads that
// every attempt waits for and registers they sit in.  (Continued traces, CONT, are
// always of one camera.)  Descriptor in memory / in the parameters: 2048^2 FP64 31.7 /
// 31.5 ms, 2048^2 mixed 21.1 / 20.1 ms, 1279x717 mixed 6.2 / 5.85 ms, the 1536^2 frame
// with the sky 30.9 / 28.8 ms.
template <int BLOCK, bool MIXED, bool ROLLED, int PASS = PASS_SINGLE, int CONT = 0, int WARPS = 12,
          bool ONE = (CONT != 0)>
__global__ void __launch_bounds__(BLOCK, 32 * WARPS / BLOCK) trace_kernel_t(const __grid_constant__ TraceArgs args) {
    __shared__ Cold<BLOCK> S;
    __shared__ KStore<ROLLED ? BLOCK : 1> K;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    constexpr bool FAR_PASS = (PASS == PASS_FAR);
    constexpr bool NEAR_PASS = (PASS == PASS_NEAR);
    static_assert(!FAR_PASS || MIXED, "the far pass runs the FP32 stages");
    static_assert(!NEAR_PASS || !MIXED, "the near pass runs FP64 stages");
    // rays of this launch: pixels (single kernel; the first far pass, but for the holes
    // of its list) or queue entries
    // (later passes; the single kernel as the critical pass of a two-pass launch)
    auto bundle = [&args](uint32_t i) -> const BundleDesc* {
        if constexpr (ONE) return &args.one;
        else return args.bundles + i;
    };
    const bool from_queue =
        (PASS == PASS_SINGLE) ? (args.in_queue != nullptr) : !(FAR_PASS && args.from_pixels != 0);
    const uint64_t total = from_queue ? static_cast<uint64_t>(*args.in_count) : args.total_rays;

    // the rounds after a ray's last pass find their queues empty (5 of the 9 launches of
    // an ordinary image): out at once, before the claims and counters (13 / 5 us each)
    if (from_queue && total == 0) return;

    // hot lane state
    double y[6], k1[6];
    double r = 0.0, h = 0.0;
    float lnp = 0.0f;  // log2 of the previous error (PI30 history)
    uint32_t acc = 0, rej = 0, flags = 0, bidx = 0;
    int mode = MODE_IDLE, wind = 0, can_early = 0;
    bool has_hist = false;
    bool critical = false;  // mixed mode: a near-critical ray (FP64 from its first step)
    float tol_sc = 1.0f;    // tolerance factor of the ray (critical_tol_scale for near-critical rays)
    bool k1_fp32 = false;  // k1 came from an FP32 far-zone stage (mixed mode)
    // A ray's end (record, pixel, invariants: atan2, the threshold root) is about as
    // long as a step attempt, and rays of a warp end one or two at a time.  The lane
    // keeps its last step instead (y, k1, h in place, y5 and k7 in local memory) and
    // waits; the warp writes all of its ends together when it refills.  Measured with
    // the lanes ending at once / together: 2048^2 FP64 38.5 / 37.0 ms, 512^2 FP64
    // 2.98 / 2.58 ms, 2048^2 mixed 27.2 / 25.2 ms.
    uint32_t end_kind = 0;  // class of the end, plus END_STEP when end_step holds the last step's end
    double end_step_mem[12];
    double* end_step = end_step_mem;
    asm volatile("" : "+l"(end_step));  // addressed memory, not twelve more register pairs
    uint32_t guard = 0;    // loop iterations spent on the current ray
    uint32_t n_cross = 0;  // disk crossings so far (translucent-disk continuation)
    uint64_t ray = 0;        // launch index of the lane's ray
#pragma unroll
    for (int i = 0; i < 6; ++i) y[i] = k1[i] = 0.0;

    // warp-uniform claim state: rays [chunk_next, chunk_end) belong to this warp
    bool queue_open = true;
    uint64_t chunk_next = 0, chunk_end = 0;
    uint32_t n_att = 0, n_acc = 0, n_rays = 0, n_rhs = 0, n_far = 0;

    for (;;) {
        if constexpr (PASS != PASS_SINGLE) {
            // park the lanes whose rays go to the other pass, and the disk hits for
            // the finish pass (one atomic per warp and queue)
            const unsigned pmask = __ballot_sync(FULL, mode == MODE_PARK);
            const unsigned fmask = __ballot_sync(FULL, mode == MODE_FINISHQ);
            if (pmask | fmask) {
                uint32_t pbase = 0, fbase = 0;
                if (pmask) {
                    const int leader = __ffs(pmask) - 1;
                    if (lane == leader) pbase = atomicAdd(args.out_count, static_cast<uint32_t>(__popc(pmask)));
                    pbase = __shfl_sync(FULL, pbase, leader);
                }
                if (fmask) {
                    const int leader = __ffs(fmask) - 1;
                    if (lane == leader) fbase = atomicAdd(args.finish_count, static_cast<uint32_t>(__popc(fmask)));
                    fbase = __shfl_sync(FULL, fbase, leader);
                }
                if (mode == MODE_PARK || mode == MODE_FINISHQ) {
                    if (mode == MODE_PARK)
                        args.out_queue[pbase + static_cast<uint32_t>(__popc(pmask & lt_mask))] = static_cast<uint32_t>(ray);
                    else
                        args.finish_queue[fbase + static_cast<uint32_t>(__popc(fmask & lt_mask))] =
                            static_cast<uint32_t>(ray);
                    double xch[7];
#pragma unroll
                    for (int i = 0; i < 6; ++i) xch[i] = y[i];
                    xch[6] = h;
                    const uint32_t misc = (has_hist ? PM_HAS_HIST : 0u) |
                                          (static_cast<uint32_t>(can_early + 1) << PM_EARLY_SHIFT) |
                                          (n_cross << PM_CROSS_SHIFT);
                    const uint32_t uch[PU_COUNT] = {acc, rej, flags, guard, static_cast<uint32_t>(wind), misc,
                                                    __float_as_uint(lnp)};
                    park_ray(args.park, ray, S, tid, xch, uch);
                    mode = MODE_IDLE;
                }
            }
        }
        {
            // ---- the ends waiting in this warp, all together, when it can refill or
            //      has nothing else to do ----
            const unsigned ended = __ballot_sync(FULL, mode == MODE_ENDED);
            const int n_free = __popc(__ballot_sync(FULL, mode == MODE_IDLE) | ended);
            if (ended && (n_free == 32 || ((queue_open || chunk_next < chunk_end) &&
                                           n_free >= static_cast<int>(args.refill_threshold)))) {
                if (mode == MODE_ENDED) {
                    const BundleDesc* Be = bundle(bidx);
                    const uint32_t cls = end_kind & 15u;
                    double target = 0.0, xch[24];
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        xch[i] = y[i];
                        xch[6 + i] = k1[i];
                    }
                    if (end_kind & END_STEP) {
#pragma unroll
                        for (int i = 0; i < 12; ++i) xch[12 + i] = end_step[i];
                        target = (cls == RT_RAY_ESCAPED)                   ? Be->r_esc
                                 : (flags & RT_RAYFLAG_EARLY_CAPTURE) != 0 ? Be->r_early
                                                                           : Be->r_capture;
                    }
                    if (cls == RT_RAY_DISK) {
                        const double rr = sqrt(bl_r2(xch[12], xch[13], xch[14], Be->a * Be->a));
                        finish_ray(Be, S, tid, RT_RAY_DISK, flags, acc, rej, wind, 0.0, 0.0, rr,
                                   disk_redshift(Be->m, Be->a, rr, S.lz0[tid]), args.out, xch);
                    } else {
                        end_ray<(CONT != 0)>(args, Be, S, tid, n_cross, cls, flags, acc, rej, wind, target, h, xch);
                        if constexpr (CONT == 3) {
                            const uint64_t local = S.local[tid];
                            args.cont.lz[Be->out_offset + local] = S.lz0[tid];
                            __threadfence();  // the chain before its length
                            *static_cast<volatile uint32_t*>(args.path.points + local) =
                                static_cast<uint32_t>(S.rit[tid] & ~kPathGap);
                        }
                    }
                    mode = MODE_IDLE;
                }
                __syncwarp();
            }
        }
        // ---- refill idle lanes: from the warp's chunk, then from a new chunk
        //      of `claim` consecutive rays (one global atomic per chunk) ----
        const unsigned idle = __ballot_sync(FULL, mode == MODE_IDLE);
        const int n_idle = __popc(idle);
        if ((queue_open || chunk_next < chunk_end) && n_idle > 0 &&
            (n_idle >= static_cast<int>(args.refill_threshold) || n_idle == 32)) {
            const uint64_t avail = chunk_end - chunk_next;
            uint64_t base2 = 0;
            bool got2 = false;
            if (avail < static_cast<uint64_t>(n_idle) && queue_open) {
                const int leader = __ffs(idle) - 1;
                unsigned long long b = 0;
                if (lane == leader) b = atomicAdd(args.queue, static_cast<unsigned long long>(args.claim));
                b = __shfl_sync(FULL, b, leader);
                if (b >= total) {
                    queue_open = false;
                } else {
                    base2 = b;
                    got2 = true;
                    if (b + args.claim >= total) queue_open = false;
                }
            }
            const uint64_t used_old = (avail < static_cast<uint64_t>(n_idle)) ? avail : n_idle;
            if (mode == MODE_IDLE) {
                const uint64_t rank = static_cast<uint64_t>(__popc(idle & lt_mask));
                uint64_t rid = ~0ull;
                if (rank < avail) rid = chunk_next + rank;
                else if (got2) rid = base2 + (rank - avail);
                uint64_t rix = rid;
                if (rid < total && (PASS != PASS_SINGLE || from_queue)) rix = args.in_queue[rid];
                if (rid < total && !(FAR_PASS && rix == kListHole)) {
                    // bundle of this ray: last bundle whose ray_begin <= rix
                    uint32_t lo = 0, hi = ONE ? 1u : args.n_bundles;
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (args.bundles[mid].ray_begin <= rix) lo = mid; else hi = mid;
                    }
                    const BundleDesc* Bc = bundle(lo);
                    bidx = lo;
                    ray = rix;
                    bool resumed = false;
                    if constexpr (PASS != PASS_SINGLE) {
                        if (from_queue) {
                            double xch[13];
                            uint32_t uch[PU_COUNT];
                            r = resume_ray(Bc, args.park, rix, rix - Bc->ray_begin,
                                                  S, tid, xch, uch);
#pragma unroll
                            for (int i = 0; i < 6; ++i) {
                                y[i] = xch[i];
                                k1[i] = xch[6 + i];
                            }
                            h = xch[12];
                            acc = uch[PU_ACC];
                            rej = uch[PU_REJ];
                            flags = uch[PU_FLAGS];
                            guard = uch[PU_GUARD];
                            wind = static_cast<int>(uch[PU_WIND]);
                            has_hist = (uch[PU_MISC] & PM_HAS_HIST) != 0u;
                            can_early = static_cast<int>((uch[PU_MISC] >> PM_EARLY_SHIFT) & 3u) - 1;
                            if constexpr (CONT != 0) n_cross = (uch[PU_MISC] >> PM_CROSS_SHIFT) & 31u;
                            lnp = __uint_as_float(uch[PU_LNP]);
                            k1_fp32 = false;
                            mode = MODE_STEP;
                            ++n_rhs;
                            resumed = true;
                        }
                    }
                    if (!resumed) {
                        double xch[12];
                        const InitResult ir =
                            init_ray(Bc, rix - Bc->ray_begin, S, tid, xch);
#pragma unroll
                        for (int i = 0; i < 6; ++i) {
                            y[i] = xch[i];
                            k1[i] = xch[6 + i];
                        }
                        r = ir.r;
                        can_early = ir.can_early;
                        h = -Bc->h0;
                        lnp = 0.0f;
                        has_hist = false;
                        acc = rej = flags = 0;
                        wind = Bc->wind0;
                        if constexpr (CONT == 3) S.rit[tid] = S.side[tid] = 0;  // points stored, page
                        k1_fp32 = false;
                        guard = 0;
                        n_cross = 0;
                        critical = false;
                        tol_sc = 1.0f;
                        // the distance of the ray's constants from the critical curve: the
                        // critical pass grades its tolerance with it; in the single mixed
                        // kernel it decides whether the ray is near-critical (the two-pass
                        // tracer's list is sorted out before); the Carter early capture
                        // takes the same value
                        if ((MIXED && !FAR_PASS && Bc->critical_band > 0.0f) ||
                            (PASS == PASS_SINGLE && !MIXED && CONT < 2 && from_queue)) {
                            const double db = shadow_distance(Bc->m, Bc->a, 0.0, Bc->rh, S.lz0[tid], S.q0[tid]);
                            if (can_early < 0) can_early = db > kEarlyCaptureMargin;
                            const double band = static_cast<double>(Bc->critical_band) * Bc->m;
                            critical = fabs(db) < band;
                            if (critical) tol_sc = critical_tol_scale(db, band);
                            if (!MIXED) ++n_rhs;  // the list's
                        }
                        mode = MODE_STEP;
                        if (!(CONT == 2 && from_queue)) ++n_rays;  // else counted by the trace that ran out of pages
                        ++n_rhs;
                    }
                }
            }
            if (got2) {
                chunk_next = base2 + (static_cast<uint64_t>(n_idle) - used_old);
                chunk_end = base2 + args.claim;
                if (chunk_end > total) chunk_end = total;
            } else {
                chunk_next += used_old;
            }
        }
        if (__ballot_sync(FULL, mode != MODE_IDLE) == 0) {
            if (!queue_open && chunk_next >= chunk_end) break;
            continue;
        }
        // mixed mode: the warp takes an FP32 far-zone step only when no stepping
        // lane is inside the FP64 zone (one instruction stream per iteration;
        // lanes in a root solve always run FP64)
        bool far = false;
        if constexpr (FAR_PASS) {
            far = true;  // near-zone rays were parked for the near pass
        } else if constexpr (MIXED) {
            const bool stepping = (mode == MODE_STEP || mode == MODE_REDO);
            const BundleDesc* Bz = bundle(bidx);
            const bool lane_far = stepping && !critical && r >= Bz->fp64_radius && r < kFp32MaxRadius;
            // every lane executes the ballot (no short-circuit around a full-mask sync)
            const unsigned near_lanes = __ballot_sync(FULL, stepping && !lane_far);
            far = lane_far && near_lanes == 0u;
        }
        if (mode == MODE_IDLE || mode == MODE_ENDED) continue;

        const BundleDesc* Bp = bundle(bidx);
        const double M = Bp->m, a = Bp->a;
        // backstop: a ray needs at most 62 iterations per attempt (attempt, <= 60
        // root iterations, redo); past that bound it is ended as unfinished
        if (++guard > 64u * Bp->max_steps + 64u) {
            flags |= RT_RAYFLAG_MAX_STEPS;
            end_kind = RT_RAY_UNFINISHED;
            mode = MODE_ENDED;
            continue;
        }
        double hh = h;
        if (mode == MODE_STEP) {
            // the initial point may already be outside the integration domain
            uint32_t term = 0;
            if (r < Bp->r_capture) term = RT_RAY_CAPTURED;
            else if (r > Bp->r_esc) term = RT_RAY_ESCAPED;
            else if (acc + rej >= Bp->max_steps) {
                flags |= RT_RAYFLAG_MAX_STEPS;
                term = RT_RAY_UNFINISHED + 16;
            }
            if (term == 0) {
                const double cap = Bp->cap_c * fmax(r - Bp->rh, 0.01 * M);
                if (fabs(h) > cap) h = -cap;
                hh = h;
                if (fabs(hh) < 1e-8) {
                    flags |= RT_RAYFLAG_STEP_UNDERFLOW;
                    term = RT_RAY_CAPTURED;
                }
            }
            if (term) {
                end_kind = term & 15u;
                mode = MODE_ENDED;
                continue;
            }
            if constexpr (FAR_PASS) {
                if (r < Bp->fp64_radius || r >= kFp32MaxRadius) {  // into the FP64 zone
                    mode = MODE_PARK;
                    continue;
                }
            }
            if constexpr (NEAR_PASS) {
                if (args.allow_exit != 0u && r >= kNearExitFactor * Bp->fp64_radius &&
                    r < kFp32MaxRadius) {  // back out of the FP64 zone
                    mode = MODE_PARK;
                    continue;
                }
            }
        } else if (mode == MODE_ROOT) {
            const double lo = S.lo[tid], hi = S.hi[tid], flo = S.flo[tid], fhi = S.fhi[tid];
            double t = (lo * fhi - hi * flo) / (fhi - flo);
            if (!(t > lo && t < hi)) t = 0.5 * (lo + hi);
            S.troot[tid] = t;
            hh = t * h;
        }

        // ---- Dormand-Prince stages 2..7 (rk45_adaptive.hpp:210-252); stage 7 is
        //      the FSAL stage at the 5th-order solution y5.  kA holds k2 for
        //      stages 3..6, then k7; est holds |h| |sum_j e_j k_j| per component. ----
        double dense5[6];  // h sum_j D_j k_j of a step that crosses z = 0 (two-pass tracer)
        double kA[6], y5[6], est[6];
        double r5 = 0.0, hf5 = 0.0, s5 = 0.0;
        const bool root = (mode == MODE_ROOT);
        if (far) {
            // FP32 radius, H and s of the FSAL stage: the projection then holds
            // H = 0 to the FP32 stages' own accuracy
            float r7, hf7, s7;
            mixed_stages(y, k1, hh, M, a, y5, kA, est, r7, hf7, s7, dense5);
            r5 = r7;
            hf5 = hf7;
            s5 = s7;
            if (mode == MODE_STEP) ++n_far;
        } else if constexpr (!FAR_PASS) {
            if constexpr (MIXED) {
                if (k1_fp32) {  // entering the FP64 zone: first stage again in FP64
                    double hf, sv;
                    ks_rhs(y, M, a, k1, hf, sv);
                    k1_fp32 = false;
                    ++n_rhs;
                }
            }
            if constexpr (ROLLED) {
                fp64_stages_rolled<BLOCK>(y, k1, hh, M, a, K, tid, root, y5, kA, est, r5, hf5, s5);
            } else {
                fp64_stages<true, NEAR_PASS>(y, k1, hh, M, a, root, y5, kA, est, dense5, r5, hf5, s5);
                const double probe = root ? y5[2] : est[2];
                // a stage left the fast forms' range (or the state is NaN), or may have unnoticed
                if (probe != probe || !(Bp->flags & BF_FAST_RANGE)) {
                    double io[39];
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        io[i] = y[i];
                        io[6 + i] = k1[i];
                    }
                    fp64_stages_special<NEAR_PASS>(io, hh, M, a, root);
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        y5[i] = io[12 + i];
                        kA[i] = io[18 + i];
                        est[i] = io[24 + i];
                        dense5[i] = io[30 + i];
                    }
                    r5 = io[36];
                    hf5 = io[37];
                    s5 = io[38];
                }
            }
        }
        n_rhs += root ? 5 : 6;

        if (PASS == PASS_SINGLE && root) {
            const double ft = y5[2];
            const int rit = ++S.rit[tid];
            const double lo = S.lo[tid], hi = S.hi[tid];
            const bool done = (ft == 0.0) || (fabs(hi - lo) < 1e-15) ||
                              (fabs(ft) < 1e-13 * (1.0 + fabs(y5[0]) + fabs(y5[1]))) || (rit >= 60);
            if (done) {
                const double rr = sqrt(bl_r2(y5[0], y5[1], y5[2], a * a));
                if (rr >= Bp->r_in && rr <= Bp->r_out && rr > Bp->rh * 1.02) {
                    // lambda at the root, one rounding in every kernel variant
                    const double lambda_step = S.lambda[tid];
                    S.lambda[tid] = fma(S.troot[tid], h, lambda_step);
                    if constexpr (CONT == 0) {
#pragma unroll
                        for (int i = 0; i < 6; ++i) end_step[i] = y5[i];
                        end_kind = RT_RAY_DISK | END_STEP;
                        mode = MODE_ENDED;
                    } else {
                        if (n_cross == 0) {
                            double xch[18];
#pragma unroll
                            for (int i = 0; i < 6; ++i) {
                                xch[i] = y[i];
                                xch[12 + i] = y5[i];
                            }
                            finish_ray(Bp, S, tid, RT_RAY_DISK, flags, acc, rej, wind, 0.0, 0.0, rr,
                                       disk_redshift(M, a, rr, S.lz0[tid]), args.out, xch);
                        }
                        mode = MODE_IDLE;
                        // translucent disk: record the crossing and go on through it
                        record_crossing(args, Bp, S, tid, n_cross, y5);
                        ++n_cross;
                        if (n_cross < kMaxCrossings) {
                            S.lambda[tid] = lambda_step;
                            mode = MODE_REDO;  // the full step again, accepted as it stands
                        } else {
                            end_continuation(args, Bp, S, tid, n_cross, RT_RAY_UNFINISHED, y5);
                        }
                    }
                } else {
                    mode = MODE_REDO;  // not on the disk: take the full step again
                }
            } else {
                const double t = S.troot[tid];
                const int side = S.side[tid];
                if ((ft > 0.0) == (S.fhi[tid] > 0.0)) {
                    S.hi[tid] = t;
                    S.fhi[tid] = ft;
                    if (side == -1) S.flo[tid] *= 0.5;
                    S.side[tid] = -1;
                } else {
                    S.lo[tid] = t;
                    S.flo[tid] = ft;
                    if (side == 1) S.fhi[tid] *= 0.5;
                    S.side[tid] = 1;
                }
            }
            continue;
        }

        // error norm (rk45_adaptive.hpp:254-261) in FP64 in every mode (in the
        // far pass on the FP32 stages' estimate); kA holds k7
        double err;
        {
            double num = 0.0, den = 1.0;
            const double rtol = Bp->rtol * static_cast<double>(tol_sc), atol = Bp->atol * static_cast<double>(tol_sc);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const double sc = rtol * fmax(fabs(y[i]), fabs(y5[i])) + atol;
                if (est[i] * den > num * sc) {
                    num = est[i];
                    den = sc;
                }
            }
            err = num / den;
        }
        if (!(err <= 1e300)) err = 1e300;  // non-finite trial: reject with the largest cut

        if (mode == MODE_STEP) {
            ++n_att;
            if (err > 1.0) {
                // reject (rk45_adaptive.hpp:303-311)
                ++rej;
                const float le = __log2f(fmaxf(static_cast<float>(err), 1e-12f));
                const float factor = pi30_factor(le, has_hist ? lnp : le, 4.0f);
                lnp = le;
                has_hist = true;
                h = -fabs(h) * clampd(0.9 * static_cast<double>(factor), 0.1, 0.9);
                continue;
            }
            ++acc;
            ++n_acc;
            bool finite = true;
#pragma unroll
            for (int i = 0; i < 6; ++i) finite = finite && isfinite(y5[i]);
            if (!finite) {
                flags |= RT_RAYFLAG_NONFINITE;
                end_kind = RT_RAY_CAPTURED;
                mode = MODE_ENDED;
                continue;
            }
            if ((Bp->flags & BF_DISK) && y[2] * y5[2] <= 0.0 && y[2] != y5[2]) {
                const double sl = y[2] / (y[2] - y5[2]);
                const double xe = y[0] + sl * (y5[0] - y[0]);
                const double ye = y[1] + sl * (y5[1] - y[1]);
                const double re = sqrt(fmax(xe * xe + ye * ye - a * a, 0.0));
                const double margin = 0.05 * re + 0.5 * M;
                if (re >= Bp->r_in - margin && re <= Bp->r_out + margin) {
                    if constexpr (PASS != PASS_SINGLE) {
                        // FP64 root on the step's dense output (its correction term from
                        // this step's stages: FP32 in the far pass, FP64 in the near
                        // pass); off the disk the step is accepted as it is
                        double xr[18];
                        const double t = dense_disk_root(y, k1, y5, kA, dense5, hh, xr + 12);
                        const double rr = sqrt(bl_r2(xr[12], xr[13], xr[14], a * a));
                        if (rr >= Bp->r_in && rr <= Bp->r_out && rr > Bp->rh * 1.02) {
                            const int wroot = wind + branch_winding(y[0], y[1], xr[12], xr[13]);
                            if constexpr (!CONT) {
                                // a disk hit: park the root point (r_hit in the step slot) for
                                // the finish pass, which writes the record in lockstep
                                S.lambda[tid] = fma(t, hh, S.lambda[tid]);
                                wind = wroot;
#pragma unroll
                                for (int i = 0; i < 6; ++i) y[i] = xr[12 + i];
                                h = rr;
                                mode = MODE_FINISHQ;
                                continue;
                            }
                            // translucent disk: the first hit's record now, the crossing
                            // recorded, and the step accepted as it stands
                            if (n_cross == 0) {
                                // finish_ray takes the root point in xr[0..5] and xr[12..17]
#pragma unroll
                                for (int i = 0; i < 6; ++i) xr[i] = xr[12 + i];
                                const double lambda_step = S.lambda[tid];
                                S.lambda[tid] = fma(t, hh, lambda_step);
                                finish_ray(Bp, S, tid, RT_RAY_DISK, flags, acc, rej, wroot, 0.0, 0.0, rr,
                                           disk_redshift(M, a, rr, S.lz0[tid]), args.out, xr);
                                S.lambda[tid] = lambda_step;
                            }
                            record_crossing(args, Bp, S, tid, n_cross, xr + 12);
                            ++n_cross;
                            if (n_cross >= kMaxCrossings) {
                                end_continuation(args, Bp, S, tid, n_cross, RT_RAY_UNFINISHED, xr + 12);
                                mode = MODE_IDLE;
                                continue;
                            }
                        }
                    } else {
                        mode = MODE_ROOT;
                        S.lo[tid] = 0.0;
                        S.flo[tid] = y[2];
                        S.hi[tid] = 1.0;
                        S.fhi[tid] = y5[2];
                        S.side[tid] = 0;
                        S.rit[tid] = 0;
                        continue;
                    }
                }
            }
        }
        // accept, second half (also the REDO of a crossing off the disk)
        mode = MODE_STEP;
        {
            // capture / escape / certain capture inside this step: the terminal point is
            // interpolated to the threshold radius, independent of where the step ended
            uint32_t term = 0;
            if (r5 < Bp->r_capture) {
                term = RT_RAY_CAPTURED;
            } else if (r5 > Bp->r_esc) {
                term = RT_RAY_ESCAPED;
            } else if (can_early != 0 && r5 < Bp->r_early) {
                if (can_early < 0)  // Carter test, once per ray, when first inside r_early
                    can_early = shadow_distance(M, a, 0.0, Bp->rh, S.lz0[tid], S.q0[tid]) > kEarlyCaptureMargin;
                // dr_BL/dlambda (kerr_invariants.hpp:140); the trace runs towards
                // decreasing lambda, so dr/dlambda > 0 means inwards
                const double rr2 = r5 * r5, z = y5[2];
                const double drdl = (rr2 * r5 * (y5[0] * kA[0] + y5[1] * kA[1]) + r5 * (rr2 + a * a) * z * kA[2]) /
                                    (rr2 * rr2 + a * a * z * z);
                if (can_early > 0 && drdl > 0.0) {
                    term = RT_RAY_CAPTURED;
                    flags |= RT_RAYFLAG_EARLY_CAPTURE;
                }
            }
            if (term) {
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    end_step[i] = y5[i];
                    end_step[6 + i] = kA[i];
                }
                end_kind = term | END_STEP;
                mode = MODE_ENDED;
                continue;
            }
        }
        {
            // projection onto H = 0 (closest root, rk45_adaptive.hpp:126-134); n = dx/dl = k7[0..2],
            // k.n and |n|^2 from |k| = 1
            double* p = y5 + 3;
            const double pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
            const double res = 0.5 * (pp - 1.0 - 2.0 * hf5 * s5 * s5);
            S.dH[tid] = fmax(S.dH[tid], fabs(res));
            if (fabs(res) >= Bp->proj_tol) {
                const double hs = hf5 * s5;
                const double kn = (s5 - 1.0) - 2.0 * hs;
                const double pn = pp - 2.0 * hs * (s5 - 1.0);
                const double nn = pp - 4.0 * hs * (s5 - 1.0) + 4.0 * hs * hs;
                const double qa = 0.5 * (nn - 2.0 * hf5 * kn * kn);
                const double qb = pn - 2.0 * hs * kn;
                const double disc = qb * qb - 4.0 * qa * res;
                if (disc >= 0.0) {
                    const double q = -0.5 * (qb + copysign(sqrt(disc), qb));
                    if (q != 0.0) {
                        const double alpha = res / q;
                        p[0] += alpha * kA[0];
                        p[1] += alpha * kA[1];
                        p[2] += alpha * kA[2];
                    }
                }
            }
        }
        if constexpr (CONT == 3) {
            // hydro model 2: the step's end, for the sampling pass
            if (fmax(r, r5) < args.path.skip) {
                S.rit[tid] |= kPathGap;
            } else {
                const double ends[6] = {y[0], y[1], y[2], y5[0], y5[1], y5[2]};
                if (!store_path_points(args, S, tid, ray, acc, rej, ends)) {
                    mode = MODE_IDLE;  // out of pages: traced again from the start
                    continue;
                }
            }
        }
        if constexpr (CONT == 2) {
            // hydro model 2: the step's chord through the Fishbone-Moncrief torus
            // (software_compute_engine.hpp:1725-1731)
            double from[3], to[3];
            bl_cartesian(y, a, from);
            bl_cartesian(y5, a, to);
            fm_segment(*args.cont.shade, from, to, S.lz0[tid],
                       args.cont.vol + (Bp->out_offset + S.local[tid]) * VL_COUNT);
        }
        wind += branch_winding(y[0], y[1], y5[0], y5[1]);
        S.lambda[tid] += hh;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            y[i] = y5[i];
            k1[i] = kA[i];
        }
        r = r5;
        if constexpr (MIXED) k1_fp32 = far;
        float factor = 5.0f;
        if (err != 0.0) {
            const float le = __log2f(fmaxf(static_cast<float>(err), 1e-12f));
            factor = pi30_factor(le, has_hist ? lnp : le, 5.0f);
            lnp = le;
            has_hist = true;
        }
        const double ah = fabs(h) * clampd(0.9 * static_cast<double>(factor), 0.2, 5.0);
        h = -clampd(ah, 1e-8, 1e13);
    }

    // warp-reduced counters (per-lane counts fit 32 bits; the sums are 64-bit)
    unsigned long long w_att = n_att, w_acc = n_acc, w_rays = n_rays, w_rhs = n_rhs, w_far = n_far;
    for (int off = 16; off > 0; off >>= 1) {
        w_att += __shfl_down_sync(FULL, w_att, off);
        w_acc += __shfl_down_sync(FULL, w_acc, off);
        w_rays += __shfl_down_sync(FULL, w_rays, off);
        w_rhs += __shfl_down_sync(FULL, w_rhs, off);
        w_far += __shfl_down_sync(FULL, w_far, off);
    }
    if (lane == 0 && w_rhs != 0) {
        if (w_rays) atomicAdd(args.stats + ST_RAYS, w_rays);
        atomicAdd(args.stats + ST_ATTEMPTS, w_att);
        atomicAdd(args.stats + ST_ACCEPTED, w_acc);
        atomicAdd(args.stats + ST_RHS, w_rhs);
        if (w_att != w_far) atomicAdd(args.stats + ST_FP64_ATTEMPTS, w_att - w_far);
    }
    if constexpr (CONT == 3) sample_ended_paths(args);
}

// The trace of a small torus-shaded frame is bound by its longest rays' chains of steps
// (3,700 where the mean is 320): 8 warps per SM, whose steps take less time.  A large one
// is bound by throughput: 12.  Near the largest spin the rays that plunge take several
// times the steps, and the line lies higher.  Measured at 12 / 8 (ms), each at
// inclinations of 80, 60 and 17 degrees:
//   320x180 (389 rays an SM)  spin 0.9   5.2/4.3    5.4/4.9    8.0/8.8
//                                  0.99  8.9/7.9    7.8/6.9   10.0/9.1
//   480x270 (876)             spin 0.9   6.8/5.8    6.2/6.9   15.4/16.0
//                                  0.99  9.5/8.0    9.2/7.7   15.1/16.3
//   640x360 (1557)            spin 0.9   8.0/8.6    8.9/9.3   25.0/26.0
//                                  0.98 10.6/10.3  10.3/9.7   24.9/25.7
//                                  0.99 12.6/10.9  12.1/10.6  24.6/25.6
//   853x480 (2766)            spin 0.9  13.0/13.8  13.7/13.8  42.2/42.9
//                                  0.99 17.5/17.4  14.1/16.3  42.4/43.3
// Spins 0 and 0.6 at 500 rays an SM 3.8/3.6 and 5.2/4.9, at 1,000 5.6/6.1 and 6.5/7.3;
// spin 0.998 at 2,000 22.4/18.5.
constexpr uint64_t kTorusLeanRaysPerSm = 640, kTorusLeanRaysPerSmExtremal = 2048;
constexpr double kTorusExtremalSpin = 0.98;
constexpr uint32_t kSampleBlock = 64;

// unshaded launches (CONT = 0), shaded ones that follow rays through the
// translucent disk (CONT = 1) and, for hydro model 2, the FP64 tracer that
// gathers the Fishbone-Moncrief torus's light step by step (CONT = 2) or stores the
// steps' points for the sampling pass (CONT = 3)
template __global__ void trace_kernel_t<64, false, false>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<256, false, false>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 0, 16>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 0, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 1, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR, 0, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR, 1, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR, 0, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR, 1, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 0, 8, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 0, 12, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 0, 16, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR, 0, 8, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR, 0, 12, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR, 0, 8, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR, 0, 12, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, false, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, true, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, true>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, true, false, PASS_FAR>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, false, false, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<256, false, false, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, false, true, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, true, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, true, true, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, true, PASS_SINGLE, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 2>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 3, 8>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_SINGLE, 3, 12>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<64, true, false, PASS_FAR, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, true, false, PASS_FAR, 1>(const __grid_constant__ TraceArgs);
template __global__ void trace_kernel_t<128, false, false, PASS_NEAR, 1>(const __grid_constant__ TraceArgs);

namespace {
// Mixed precision always uses the rolled FP64 step (its FP64 steps are a
// minority; the rolled form keeps the loop small).  Rolled kernels exist for
// 64- and 128-thread blocks (their stage store is 36 KB of shared memory at 128).
template <int CONT>
const void* kernel_for_t(uint32_t block, bool mixed, bool rolled) {
    if (mixed) {
        return (block == 64) ? reinterpret_cast<const void*>(&trace_kernel_t<64, true, true, PASS_SINGLE, CONT>)
                             : reinterpret_cast<const void*>(&trace_kernel_t<128, true, true, PASS_SINGLE, CONT>);
    }
    if (rolled) {
        return (block == 64) ? reinterpret_cast<const void*>(&trace_kernel_t<64, false, true, PASS_SINGLE, CONT>)
                             : reinterpret_cast<const void*>(&trace_kernel_t<128, false, true, PASS_SINGLE, CONT>);
    }
    switch (block) {
        case 64: return reinterpret_cast<const void*>(&trace_kernel_t<64, false, false, PASS_SINGLE, CONT>);
        case 256: return reinterpret_cast<const void*>(&trace_kernel_t<256, false, false, PASS_SINGLE, CONT>);
        default: return reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, CONT>);
    }
}

const void* kernel_for(uint32_t block, bool mixed, bool rolled, int cont = 0) {
    if (cont == 2) return reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 2>);
    return (cont == 1) ? kernel_for_t<1>(block, mixed, rolled) : kernel_for_t<0>(block, mixed, rolled);
}

// The plain FP64 tracer in 128-thread blocks with 8, 12 or 16 warps per SM.
template <int WARPS>
const void* plain_kernel_t(bool cont, bool one) {
    if constexpr (WARPS < 16)
        if (cont) return reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 1, WARPS>);
    return one ? reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 0, WARPS, true>)
               : reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 0, WARPS, false>);
}

// Rays per SM from which the plain FP64 tracer takes 16 warps.  More warps raise the
// rate and lengthen one attempt, so the longest rays' tail has to be a small part of
// the launch.  12 / 16 warps, three cameras (face-on, grazing, wide view): 1448^2
// 17.2 / 16.2, 22.3 / 23.3, 12.9 / 12.4 ms; 1740^2 24.7 / 23.2, 32.8 / 34.3,
// 18.4 / 17.5; 2048^2 34.0 / 31.9, 43.4 / 42.0, 25.3 / 24.0.  The line is at 3.6 M rays.
constexpr uint64_t kWideRaysPerSm = 24576;
// Rays per SM up to which it takes 8: the rays that 12 warps hold at once.  12 / 8
// warps, the same cameras: 96^2 0.76 / 0.67, 1.43 / 1.36, 1.26 / 1.23 ms; 224^2 0.92 /
// 0.74, 1.75 / 1.54, 1.87 / 1.69; past the line 288^2 0.97 / 1.04, 1.89 / 1.70, 1.98 / 1.93.
constexpr uint64_t kLeanRaysPerSm = 384;
// The same for the passes of the mixed tracer, in rays of the whole launch (each pass
// runs a part of them): 213x119 1.00 / 0.81, 1.73 / 1.51, 2.29 / 1.99 ms; 512x288 1.39 /
// 1.33, 2.50 / 2.25, 2.56 / 2.42; past the line 768x432 2.02 / 2.05, 3.17 / 3.30, 3.36 / 3.11.
constexpr uint64_t kLeanMixedRaysPerSm = 1024;
}  // namespace

// Loads the kernels that launch_trace may pick beside those of trace_occupancy.
void preload_trace_shapes() {
    int n = 0;
    for (const void* k : {plain_kernel_t<8>(false, false), plain_kernel_t<16>(false, false)})
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 128, 0) != cudaSuccess) cudaGetLastError();
}

uint32_t kernel_block(uint32_t block, bool mixed, bool rolled) {
    if ((mixed || rolled) && block > 128) return 128;
    return block;
}

int trace_occupancy(uint32_t block, bool mixed, bool rolled) {
    int n = 0;
    block = kernel_block(block, mixed, rolled);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_for(block, mixed, rolled), static_cast<int>(block), 0) !=
        cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n;
}

// Finish pass of the two-pass mixed tracer: the record and pixel of every disk
// hit parked by the far and near passes (root point, r_hit in the step slot).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) finish_kernel_t(TraceArgs args) {
    __shared__ Cold<BLOCK> S;
    const int tid = threadIdx.x;
    const uint64_t count = *args.in_count;
    const uint64_t n = args.park.n;
    for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * BLOCK + tid; j < count;
         j += static_cast<uint64_t>(gridDim.x) * BLOCK) {
        const uint64_t ray = args.in_queue[j];
        uint32_t lo = 0, hi = args.n_bundles;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (args.bundles[mid].ray_begin <= ray) lo = mid; else hi = mid;
        }
        const BundleDesc* Bp = args.bundles + lo;
        double xch[18];
#pragma unroll
        for (int i = 0; i < 6; ++i) xch[i] = xch[12 + i] = args.park.d[(PD_Y + i) * n + ray];
        const double r_hit = args.park.d[PD_H * n + ray];
        S.lambda[tid] = args.park.d[PD_LAMBDA * n + ray];
        S.dH[tid] = args.park.d[PD_DH * n + ray];
        S.lz0[tid] = args.park.d[PD_LZ0 * n + ray];
        S.q0[tid] = args.park.d[PD_Q0 * n + ray];
        S.local[tid] = ray - Bp->ray_begin;
        finish_ray(Bp, S, tid, RT_RAY_DISK, args.park.u[PU_FLAGS * n + ray], args.park.u[PU_ACC * n + ray],
                          args.park.u[PU_REJ * n + ray], static_cast<int>(args.park.u[PU_WIND * n + ray]), 0.0, 0.0,
                          r_hit, disk_redshift(Bp->m, Bp->a, r_hit, S.lz0[tid]), args.out, xch);
    }
}
template __global__ void finish_kernel_t<128>(TraceArgs);

namespace {
template <bool MIXED, int PASS, int WARPS>
const void* pass_kernel_t(bool cont, bool one) {
    if (cont) return reinterpret_cast<const void*>(&trace_kernel_t<128, MIXED, false, PASS, 1, WARPS>);
    return one ? reinterpret_cast<const void*>(&trace_kernel_t<128, MIXED, false, PASS, 0, WARPS, true>)
               : reinterpret_cast<const void*>(&trace_kernel_t<128, MIXED, false, PASS, 0, WARPS, false>);
}

const void* pass_kernel(int pass, uint32_t block, bool lean, bool cont, bool one) {
    if (pass == PASS_FAR) {
        if (block == 64)
            return cont ? reinterpret_cast<const void*>(&trace_kernel_t<64, true, false, PASS_FAR, 1>)
                        : reinterpret_cast<const void*>(&trace_kernel_t<64, true, false, PASS_FAR, 0>);
        return lean ? pass_kernel_t<true, PASS_FAR, 8>(cont, one) : pass_kernel_t<true, PASS_FAR, 12>(cont, one);
    }
    return lean ? pass_kernel_t<false, PASS_NEAR, 8>(cont, one) : pass_kernel_t<false, PASS_NEAR, 12>(cont, one);
}

int trace_pass_occupancy(int pass, uint32_t block, bool lean) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pass_kernel(pass, block, lean, false, false), static_cast<int>(block), 0) !=
        cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n;
}

// One pass of the two-pass mixed tracer (PASS_FAR or PASS_NEAR).
void launch_trace_pass(const TraceArgs& args, int pass, uint32_t grid, uint32_t block, bool lean, cudaStream_t stream) {
    void* params[] = {const_cast<TraceArgs*>(&args)};
    cudaLaunchKernel(pass_kernel(pass, block, lean, args.cont.cross != nullptr, args.has_one != 0u), dim3(grid),
                     dim3(block), params, 0, stream);
}
}  // namespace

// The rays of a two-pass launch's band sorted out before its passes: the near-critical
// ones to the critical pass's list (with the length class when that list is sorted
// below), and a list for the first far pass that has a hole in place of each of them,
// so that its warps keep their neighbours (closed up, in the order of the blocks, the
// far pass is 2 % faster and the near pass after it 18 % slower).  The critical pass then
// runs beside the far pass, and a ray is on exactly one list.  Measured, the far pass
// sorting its rays out as it meets them and the critical pass after it / this: 213x119
// 1.75 / 1.54 ms, 2048^2 20.1 / 19.2, a table of 40 cameras 35.5 / 34.1, a burst of
// server requests 19.3 / 17.9.
__global__ void __launch_bounds__(128) band_list_kernel(const __grid_constant__ TraceArgs args, uint32_t* far_list,
                                                        uint32_t* crit_list, uint32_t* crit_count, bool classes) {
    __shared__ Cold<128> S;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * 128 + tid, rix = args.ray_base + i;
    bool critical = false;
    uint32_t cls = 0;
    if (i < args.total_rays) {
        uint32_t lo = 0, hi = args.has_one ? 1u : args.n_bundles;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (args.bundles[mid].ray_begin <= rix) lo = mid; else hi = mid;
        }
        const BundleDesc* B = args.has_one ? &args.one : args.bundles + lo;
        if (B->critical_band > 0.0f) {
            double xch[12];
            init_ray(B, rix - B->ray_begin, S, tid, xch);
            const double db = shadow_distance(B->m, B->a, 0.0, B->rh, S.lz0[tid], S.q0[tid]);
            const double band = static_cast<double>(B->critical_band) * B->m;
            critical = fabs(db) < band;
            if (critical && classes) cls = critical_class(db, band);
        }
        far_list[i] = critical ? kListHole : static_cast<uint32_t>(rix);
    }
    const unsigned crit = __ballot_sync(~0u, critical);
    uint32_t at = 0;
    if (lane == 0 && crit) at = atomicAdd(crit_count, static_cast<uint32_t>(__popc(crit)));
    at = __shfl_sync(~0u, at, 0);
    if (critical) crit_list[at + __popc(crit & ((1u << lane) - 1u))] = static_cast<uint32_t>(rix) | (cls << kCritClassShift);
}

// The near-critical list, sorted by length class.  It holds the rays in about the order
// of the launch; across the critical curve neighbours differ several times over
// in attempts (the tolerance is graded by |d_b|, and the orbits near the photon sphere
// add to it), so a warp of neighbours runs at 17 to 21 of 32 lanes.  A counting sort
// into 32 classes (two small launches) puts rays of like length in a warp and the
// longest first.  In the list's order / sorted: the 1536^2 frame with the sky 39.9 /
// 36.0 ms, a table of 40 cameras 39.6 / 36.3 ms, 1279x717 6.46 / 6.28 ms.
constexpr uint32_t kCritBlock = 256;
// Rays per SM of the launch from which the list is sorted: the launches and the pass
// between cost about 40 us of a chain that a small image waits for (213x119 1.45 /
// 1.55 ms, 320x180 1.55 / 1.56, 512x288 1.33 / 1.30 and 2.41 / 2.33).
constexpr uint64_t kCritSortRaysPerSm = 768;

__global__ void __launch_bounds__(kCritBlock) crit_count_kernel(const uint32_t* __restrict__ list,
                                                                const uint32_t* __restrict__ count,
                                                                uint32_t* __restrict__ histogram) {
    __shared__ uint32_t h[kCritClasses];
    if (threadIdx.x < kCritClasses) h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t n = *count;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kCritBlock + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * kCritBlock)
        atomicAdd(h + (list[i] >> kCritClassShift), 1u);
    __syncthreads();
    if (threadIdx.x < kCritClasses && h[threadIdx.x]) atomicAdd(histogram + threadIdx.x, h[threadIdx.x]);
}

// Rays in blocks of kCritBlock, each block's share of a class reserved with one atomic
// on the class's cursor, so that a class keeps about the order of the list.
__global__ void __launch_bounds__(kCritBlock) crit_scatter_kernel(const uint32_t* __restrict__ list,
                                                                  const uint32_t* __restrict__ count,
                                                                  const uint32_t* __restrict__ histogram,
                                                                  uint32_t* __restrict__ cursor,
                                                                  uint32_t* __restrict__ sorted) {
    __shared__ uint32_t first[kCritClasses], base[kCritClasses], taken[kCritClasses];
    if (threadIdx.x == 0) {
        uint32_t at = 0;
        for (uint32_t k = 0; k < kCritClasses; ++k) {
            first[k] = at;
            at += histogram[k];
        }
    }
    const uint64_t n = *count;
    for (uint64_t b = static_cast<uint64_t>(blockIdx.x) * kCritBlock; b < n;
         b += static_cast<uint64_t>(gridDim.x) * kCritBlock) {
        if (threadIdx.x < kCritClasses) taken[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t i = b + threadIdx.x;
        uint32_t v = 0, k = 0, rank = 0;
        if (i < n) {
            v = list[i];
            k = v >> kCritClassShift;
            rank = atomicAdd(taken + k, 1u);
        }
        __syncthreads();
        if (threadIdx.x < kCritClasses)
            base[threadIdx.x] = first[threadIdx.x] +
                                (taken[threadIdx.x] ? atomicAdd(cursor + threadIdx.x, taken[threadIdx.x]) : 0u);
        __syncthreads();
        if (i < n) sorted[base[k] + rank] = v & ((1u << kCritClassShift) - 1u);
        __syncthreads();
    }
}

// Rounds of the two-pass mixed tracer: far pass (FP32) then near pass (FP64),
// the last near pass keeping every ray to its end.  A ray typically needs one
// round (in to a disk crossing or the near zone, and out); rays left after the
// last far pass finish in FP64.
constexpr int kMixedRounds = 4;
// Refill threshold of the near pass: its rays resume from parked state (a few
// loads and one RHS), so refilling a partly idle warp is cheap, while the
// near-zone work per ray (disk root, photon-region orbits) varies widely.
constexpr uint32_t kNearRefill = 16;  // measured best of 1, 4, 8, 16, 32
// Block of the critical pass (the FP64 kernel's default shape).
constexpr uint32_t kCriticalBlock = 128;

uint64_t two_pass_state_bytes(uint64_t n) {
    return n * (sizeof(double) * PD_COUNT + sizeof(uint32_t) * PU_COUNT + 4 * sizeof(uint32_t));
}

// Per-band queue counters (kBandCounterBytes): [0] far-pass claim (u64), [8]
// near queue count (u32), [12] far queue count (u32), [16] near-pass claim
// (u64), zeroed pairwise before each pass; [24] finish queue count (u32), [32]
// near-critical list's count (u32), [40] the critical pass's claim (u64) and [64] the
// near-critical classes' histogram and cursors (kCritClasses u32 each), zeroed once.
namespace {
// A band's part of the launch's scratch.
struct Band {
    uint32_t *near_q, *far_q, *finish_q, *crit_q;
    char* counters;
    uint64_t begin, count;
};

// The band's rays sorted out (band_list_kernel): the far list in the far queue, which the
// near pass fills later; the critical list, before it is sorted, in the near queue, which
// the far pass fills.
cudaError_t enqueue_lists(TraceArgs args, const Band& band, bool sorted, int sm_count, cudaStream_t s) {
    args.total_rays = band.count;
    args.ray_base = band.begin;
    char* qb = band.counters;
    cudaError_t e = cudaMemsetAsync(qb, 0, kBandCounterBytes, s);
    if (e != cudaSuccess) return e;
    uint32_t* n_crit = reinterpret_cast<uint32_t*>(qb + 32);
    uint32_t* crit_list = sorted ? band.near_q : band.crit_q;
    band_list_kernel<<<static_cast<uint32_t>((band.count + 127) / 128), 128, 0, s>>>(
        args, band.far_q, crit_list, n_crit, sorted);
    if ((e = cudaGetLastError()) != cudaSuccess || !sorted) return e;
    uint32_t* hist = reinterpret_cast<uint32_t*>(qb + 64);
    const uint32_t blocks =
        static_cast<uint32_t>(std::min<uint64_t>((band.count + kCritBlock - 1) / kCritBlock, 2u * sm_count));
    crit_count_kernel<<<blocks, kCritBlock, 0, s>>>(crit_list, n_crit, hist);
    crit_scatter_kernel<<<blocks, kCritBlock, 0, s>>>(crit_list, n_crit, hist, hist + kCritClasses, band.crit_q);
    return cudaGetLastError();
}

cudaError_t enqueue_band(TraceArgs args, const TwoPassBuffers& buf, const Band& band, uint32_t far_grid,
                         uint32_t far_block, uint32_t near_grid, uint32_t finish_grid, int sm_count, uint32_t crit_ctas,
                         bool crit_beside, bool crit_first, bool lean, cudaStream_t s) {
    char* qb = band.counters;
    uint32_t *near_q = band.near_q, *far_q = band.far_q;
    args.park = buf.park;
    args.total_rays = band.count;
    args.ray_base = band.begin;
    args.finish_queue = band.finish_q;
    args.finish_count = reinterpret_cast<uint32_t*>(qb + 24);
    const uint32_t far_refill = args.refill_threshold;
    cudaError_t e = cudaSuccess;
    // critical pass: the near-critical rays, FP64 from their pixels to their end at
    // their graded tolerance (the single FP64 kernel over a queue); on its own stream it
    // runs beside the other passes, each filling the SMs the other's tail leaves idle.
    // In a band of several, whose gaps another band's passes fill, it comes after the
    // far pass (the 1536^2 frame 29.6 / 30.2 ms before it)
    const TraceArgs base = args;
    const auto critical_pass = [&]() -> cudaError_t {
        TraceArgs c = base;
        c.queue = reinterpret_cast<unsigned long long*>(qb + 40);
        c.refill_threshold = 32;
        c.in_queue = band.crit_q;
        c.in_count = reinterpret_cast<const uint32_t*>(qb + 32);
        c.finish_queue = nullptr;
        c.finish_count = nullptr;
        cudaStream_t cs = s;
        cudaError_t ce = cudaSuccess;
        if (crit_beside) {
            cs = static_cast<cudaStream_t>(buf.crit_stream);
            if ((ce = cudaEventRecord(static_cast<cudaEvent_t>(buf.crit_fork), s)) != cudaSuccess) return ce;
            if ((ce = cudaStreamWaitEvent(cs, static_cast<cudaEvent_t>(buf.crit_fork), 0)) != cudaSuccess) return ce;
        }
        launch_trace(c, sm_count, crit_ctas, kCriticalBlock, false, false, cs, lean);
        if ((ce = cudaGetLastError()) != cudaSuccess) return ce;
        return crit_beside ? cudaEventRecord(static_cast<cudaEvent_t>(buf.crit_join), cs) : cudaSuccess;
    };
    if (crit_first && (e = critical_pass()) != cudaSuccess) return e;
    for (int round = 0; e == cudaSuccess && round < kMixedRounds; ++round) {
        // far pass: the far list (first round) or the far queue -> near queue
        if (round > 0 && (e = cudaMemsetAsync(qb, 0, 12, s)) != cudaSuccess) break;
        args.queue = reinterpret_cast<unsigned long long*>(qb);
        args.refill_threshold = far_refill;
        args.from_pixels = (round == 0) ? 1u : 0u;
        args.allow_exit = 0;
        args.in_queue = far_q;
        args.in_count = reinterpret_cast<const uint32_t*>(qb + 12);
        args.out_queue = near_q;
        args.out_count = reinterpret_cast<uint32_t*>(qb + 8);
        launch_trace_pass(args, PASS_FAR, far_grid, far_block, lean, s);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        if (round == 0 && !crit_first && (e = critical_pass()) != cudaSuccess) break;
        // near pass: near queue -> far queue (the last one keeps its rays)
        if ((e = cudaMemsetAsync(qb + 12, 0, 12, s)) != cudaSuccess) break;
        args.queue = reinterpret_cast<unsigned long long*>(qb + 16);
        args.refill_threshold = far_refill < kNearRefill ? far_refill : kNearRefill;
        args.from_pixels = 0;
        args.allow_exit = (round + 1 < kMixedRounds) ? 1u : 0u;
        args.in_queue = near_q;
        args.in_count = reinterpret_cast<const uint32_t*>(qb + 8);
        args.out_queue = far_q;
        args.out_count = reinterpret_cast<uint32_t*>(qb + 12);
        launch_trace_pass(args, PASS_NEAR, near_grid, 128, lean, s);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    // finish pass over the band's parked disk hits
    args.in_queue = args.finish_queue;
    args.in_count = args.finish_count;
    finish_kernel_t<128><<<finish_grid, 128, 0, s>>>(args);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (crit_beside) e = cudaStreamWaitEvent(s, static_cast<cudaEvent_t>(buf.crit_join), 0);
    return e;
}
}  // namespace

int enqueue_two_pass(const TraceArgs& base, const TwoPassBuffers& buf, int sm_count, uint32_t far_block,
                     void* stream, void* stream2, void* fork, void* join, uint32_t bands, BandHook after_band,
                     void* hook_ctx) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaStream_t s2 = static_cast<cudaStream_t>(stream2);
    const uint64_t n = base.total_rays;
    if (!s2 || !fork || !join) bands = 1;
    bands = bands < 1 ? 1 : (bands > kMaxBands ? kMaxBands : bands);
    if (static_cast<uint64_t>(bands) > n) bands = static_cast<uint32_t>(n > 0 ? n : 1);
    far_block = (far_block == 64) ? 64u : 128u;
    const bool lean = far_block == 128u && n <= kLeanMixedRaysPerSm * static_cast<uint64_t>(sm_count);
    const int far_occ = trace_pass_occupancy(PASS_FAR, far_block, lean);
    const int near_occ = trace_pass_occupancy(PASS_NEAR, 128, lean);
    const uint32_t far_grid = static_cast<uint32_t>(sm_count) * static_cast<uint32_t>(far_occ > 1 ? far_occ : 1);
    const uint32_t near_grid = static_cast<uint32_t>(sm_count) * static_cast<uint32_t>(near_occ > 1 ? near_occ : 1);
    const uint32_t finish_grid = static_cast<uint32_t>(sm_count) * 8u;
    const int crit_occ = trace_occupancy(kCriticalBlock, false, false);
    const uint32_t crit_ctas = static_cast<uint32_t>(crit_occ > 1 ? crit_occ : 1);
    cudaError_t e = cudaSuccess;
    // bands of whole warps' worth of rays (multiples of 32); every band's lists first,
    // while the SMs are free
    const uint64_t per = ((n + bands - 1) / bands + 31) / 32 * 32;
    // a class needs the index's upper bits
    const bool sorted = n <= (1ull << kCritClassShift) && n > kCritSortRaysPerSm * static_cast<uint64_t>(sm_count);
    Band part[kMaxBands];
    uint32_t n_parts = 0;
    for (uint64_t begin = 0; begin < n; begin += per, ++n_parts) {
        Band& p = part[n_parts];
        p.begin = begin;
        p.count = std::min(per, n - begin);
        p.near_q = buf.queues + 4 * begin;
        p.far_q = p.near_q + p.count;
        p.finish_q = p.far_q + p.count;
        p.crit_q = p.finish_q + p.count;
        p.counters = buf.counters + kBandCounterBytes * n_parts;
        if ((e = enqueue_lists(base, p, sorted, sm_count, s)) != cudaSuccess) return static_cast<int>(e);
    }
    if (bands > 1) {
        if ((e = cudaEventRecord(static_cast<cudaEvent_t>(fork), s)) != cudaSuccess) return static_cast<int>(e);
        if ((e = cudaStreamWaitEvent(s2, static_cast<cudaEvent_t>(fork), 0)) != cudaSuccess) return static_cast<int>(e);
    }
    // a band's hook is enqueued after the next band's trace, so its work overlaps that trace
    const Band* prev = nullptr;
    cudaStream_t prev_stream = nullptr;
    const bool crit_beside = bands == 1 && buf.crit_stream && buf.crit_fork && buf.crit_join;
    for (uint32_t b = 0; b < n_parts && e == cudaSuccess; ++b) {
        cudaStream_t sb = (b & 1u) ? s2 : s;
        e = enqueue_band(base, buf, part[b], far_grid, far_block, near_grid, finish_grid, sm_count, crit_ctas, crit_beside,
                         bands == 1, lean, sb);
        if (e == cudaSuccess && after_band && prev)
            e = static_cast<cudaError_t>(after_band(hook_ctx, prev->begin, prev->count, prev_stream));
        prev = &part[b];
        prev_stream = sb;
    }
    if (e == cudaSuccess && after_band && prev)
        e = static_cast<cudaError_t>(after_band(hook_ctx, prev->begin, prev->count, prev_stream));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (bands > 1) {
        if ((e = cudaEventRecord(static_cast<cudaEvent_t>(join), s2)) != cudaSuccess) return static_cast<int>(e);
        e = cudaStreamWaitEvent(s, static_cast<cudaEvent_t>(join), 0);
    }
    return static_cast<int>(e);
}

void launch_trace(const TraceArgs& args, int sm_count, uint32_t ctas_per_sm, uint32_t block, bool mixed, bool rolled,
                  void* stream, bool lean) {
    void* params[] = {const_cast<TraceArgs*>(&args)};
    // hydro model 2: the FP64 straight-line tracer in 128-thread blocks
    const int cont = args.cont.vol ? 2 : (args.cont.cross ? 1 : 0);
    block = (cont == 2) ? 128u : kernel_block(block, mixed, rolled);
    const void* kernel = kernel_for(block, mixed, rolled, cont);
    // 8 or 16 warps per SM only where the caller left the CTAs per SM at the occupancy
    // maximum; the critical pass's rays are counted on the device, so its caller decides
    if (!mixed && !rolled && cont != 2 && block == 128u) {
        const uint64_t sm = static_cast<uint64_t>(sm_count);
        const bool one = args.has_one != 0u, shaped = ctas_per_sm >= 3u;
        kernel = plain_kernel_t<12>(cont == 1, one);
        if (shaped && (lean || (!args.in_queue && args.total_rays <= kLeanRaysPerSm * sm))) {
            kernel = plain_kernel_t<8>(cont == 1, one);
            ctas_per_sm = 2;
        } else if (shaped && cont == 0 && !args.in_queue && args.total_rays >= kWideRaysPerSm * sm) {
            kernel = plain_kernel_t<16>(false, one);
            ctas_per_sm = 4;
        }
    }
    cudaLaunchKernel(kernel, dim3(static_cast<uint32_t>(sm_count) * ctas_per_sm), dim3(block), params, 0,
                     static_cast<cudaStream_t>(stream));
}

// The order in which a torus-shaded trace takes its rays: those inside the critical
// curve first.  They plunge, and their steps shrink with the distance to the horizon
// (about 1,750 a ray against 180 for one that turns back), so that a warp of them begun
// late runs on alone; begun first, and with their like in a warp, the short rays fill in.
__global__ void __launch_bounds__(128) torus_order_kernel(const __grid_constant__ TraceArgs args) {
    __shared__ Cold<128> S;
    const BundleDesc& B = args.one;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * 128 + tid;
    const bool live = i < args.total_rays;
    bool plunges = false;
    if (live) {
        double xch[12];
        init_ray(&B, args.ray_base + i, S, tid, xch);
        plunges = shadow_distance(B.m, B.a, 0.0, B.rh, S.lz0[tid], S.q0[tid]) > 0.0;
    }
    const unsigned first = __ballot_sync(~0u, live && plunges), rest = __ballot_sync(~0u, live && !plunges);
    uint32_t at = 0;
    if (lane < 2) {
        const uint32_t n = static_cast<uint32_t>(__popc(lane == 0 ? first : rest));
        if (n) at = atomicAdd(args.path.cursor + PC_PLUNGING + lane, n);
    }
    const uint32_t at_first = __shfl_sync(~0u, at, 0), at_rest = __shfl_sync(~0u, at, 1);
    const unsigned below = (1u << lane) - 1u;
    const uint32_t total = static_cast<uint32_t>(args.total_rays);
    if (live) {
        const uint32_t to = plunges ? at_first + __popc(first & below) : total - 1u - (at_rest + __popc(rest & below));
        args.path.order[to] = static_cast<uint32_t>(args.ray_base + i);
    }
    if (i == 0) args.path.cursor[PC_TOTAL] = total;
}

// The sampling pass of a torus-shaded trace: what the trace's idle warps left of it.
__global__ void __launch_bounds__(kSampleBlock) torus_sample_kernel(const __grid_constant__ TraceArgs args) {
    const uint64_t i = (static_cast<uint64_t>(blockIdx.x) * kSampleBlock + threadIdx.x) / kPathLanes;
    uint32_t local = 0, points = 0;
    if (i < args.total_rays) {
        local = args.path.order[i];
        points = args.path.points[local];
        if (points == kPathOpen) points = 0;
    }
    if (__any_sync(0xffffffffu, points != 0)) sample_paths(args, local, points);
}

int enqueue_torus(const TraceArgs& base, int sm_count, uint32_t ctas_per_sm, char* claims, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    TraceArgs args = base;
    cudaError_t e = cudaMemsetAsync(claims, 0, 72, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(args.path.cursor, 0, kPathCursorBytes, s);
    if (e == cudaSuccess)  // no ray has ended
        e = cudaMemsetAsync(args.path.points + args.ray_base, 0xff, sizeof(uint32_t) * args.total_rays, s);
    if (e != cudaSuccess) return static_cast<int>(e);
    torus_order_kernel<<<static_cast<uint32_t>((args.total_rays + 127) / 128), 128, 0, s>>>(args);
    if ((e = cudaGetLastError()) != cudaSuccess) return static_cast<int>(e);
    args.queue = reinterpret_cast<unsigned long long*>(claims);
    args.in_queue = args.path.order;
    args.in_count = args.path.cursor + PC_TOTAL;
    void* params[] = {&args};
    const bool extremal = std::fabs(args.one.a) >= kTorusExtremalSpin * args.one.m;
    const bool lean = args.total_rays <=
                      (extremal ? kTorusLeanRaysPerSmExtremal : kTorusLeanRaysPerSm) * static_cast<uint64_t>(sm_count);
    cudaLaunchKernel(lean ? reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 3, 8>)
                          : reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 3, 12>),
                     dim3(static_cast<uint32_t>(sm_count) * std::min(ctas_per_sm, lean ? 2u : 3u)), dim3(128), params, 0,
                     s);
    if ((e = cudaGetLastError()) != cudaSuccess) return static_cast<int>(e);
    torus_sample_kernel<<<static_cast<uint32_t>((args.total_rays * kPathLanes + kSampleBlock - 1) / kSampleBlock), kSampleBlock, 0,
                          s>>>(args);
    if ((e = cudaGetLastError()) != cudaSuccess) return static_cast<int>(e);
    // the rays whose pages ran out
    args.queue = reinterpret_cast<unsigned long long*>(claims + 64);
    args.in_queue = args.path.overflow;
    args.in_count = args.path.cursor + PC_OVERFLOW;
    cudaLaunchKernel(reinterpret_cast<const void*>(&trace_kernel_t<128, false, false, PASS_SINGLE, 2>),
                     dim3(static_cast<uint32_t>(sm_count) * std::min(ctas_per_sm, 3u)), dim3(128), params, 0, s);
    return static_cast<int>(cudaGetLastError());
}

rt_launch_config resolve_launch_config(rt_launch_config c, bool mixed) {
    if (c.block_size != 64 && c.block_size != 128 && c.block_size != 256) c.block_size = 128;
    c.fp64_rolled = c.fp64_rolled ? 1u : 0u;
    c.mixed_single_kernel = c.mixed_single_kernel ? 1u : 0u;
    c.block_size = kernel_block(c.block_size, mixed, c.fp64_rolled != 0);
    const int occ = trace_occupancy(c.block_size, mixed, c.fp64_rolled != 0);
    if (c.ctas_per_sm == 0 || static_cast<int>(c.ctas_per_sm) > occ) c.ctas_per_sm = occ > 1 ? occ : 1;
    // defaults from the autotuner on B200: whole-warp refills of 32 consecutive rays
    if (c.refill_threshold == 0 || c.refill_threshold > 32) c.refill_threshold = 32;
    if (c.rays_per_thread == 0 || c.rays_per_thread > 64) c.rays_per_thread = 1;
    return c;
}

}  // namespace relsim
