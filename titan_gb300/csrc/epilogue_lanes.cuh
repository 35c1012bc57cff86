// epilogue_lanes.cuh -- the FP64 mass phase with a lane per component: a warp
// takes ten masses, component c of the warp's mass j in lane 10 c + j.
//
// For small tiles, whose masses fit a few warps, the mass phase is latency: a
// dependent FP64 operation takes 61 cycles, and three components in one
// thread queue three of them behind each other on the SM sub-partition's FP64
// unit (64 cycles a warp instruction).  Spread over lanes the components
// share each instruction, and a dot product costs shuffles instead of
// issue slots.  Products stay on the FP64 unit here (61 cycles against about
// 150 for alu_mul between packed operands); square roots and divisions are
// fp64_alu.cuh's (280 and 250 cycles against 710 and 1,700).
//
// The operations and their order are those of integrate and plane_apply
// (epilogue.cuh, step_math.cuh): the same bits.  Measured, us per step, a
// thread per mass and this: 5^3 robot in the air 5.4 -> 4.6, standing on its
// plane 8.5 -> 6.2, 9^3 7.0 -> 6.2, 14^3 8.3 -> 7.4, 20^3 12.9 -> 12.3.
#pragma once

#include "engine.h"
#include "epilogue.cuh"
#include "fp64_alu.cuh"
#include "step_math.cuh"

namespace tg {
namespace {

constexpr int kLaneMasses = 10;  // masses per warp

__device__ __noinline__ double sqrt_wide(double n) { return sqrt(n); }
__device__ __noinline__ double div_wide(double a, double b) { return a / b; }

__device__ __forceinline__ double sqrt_alu(double n) {
    uint32_t bad = 0;
    const Alu N = alu_unpack(n, bad);
    AluDivisor d;
    const double r = alu_pack(alu_sqrt(N, d));
    if (!alu_nonzero(N)) return n;
    return alu_bad(bad) || (N.se >> 31) ? sqrt_wide(n) : r;
}
__device__ __forceinline__ double div_alu(double a, double b) {
    uint32_t bad = 0;
    const Alu y = alu_unpack(b, bad);
    const double r = alu_pack(alu_div(alu_unpack(a, bad), alu_divisor(y)));
    return alu_bad(bad) || !alu_nonzero(y) ? div_wide(a, b) : r;
}

// (p0 + p1) + p2 of the mass's components
__device__ __forceinline__ double lane_sum(double p, int j) {
    const double p0 = __shfl_sync(0xffffffffu, p, j), p1 = __shfl_sync(0xffffffffu, p, kLaneMasses + j),
                 p2 = __shfl_sync(0xffffffffu, p, 2 * kLaneMasses + j);
    return (p0 + p1) + p2;
}

// The force with a contact plane's added (plane_apply); n: the normal's
// component.  want: the mass has this plane.  Called by whole warps.
__device__ __forceinline__ double plane_lanes(double n, double off, double fk, double fs, double x, double v, double F,
                                              int j, bool want) {
    const double disp = lane_sum(x * n, j) - off;
    const bool contact = want && disp < 0;
    if (!__any_sync(0xffffffffu, contact)) return F;
    double G = F;
    const double fn = n * lane_sum(F * n, j);
    if (fs > 0 || fk > 0) {
        const double vp = v - n * lane_sum(v * n, j);
        const double vn = sqrt_alu(lane_sum(vp * vp, j)), fnn = sqrt_alu(lane_sum(fn * fn, j));
        const bool moving = vn > 1e-16;
        if (__any_sync(0xffffffffu, contact && moving)) {
            const double q = div_alu(vp * (fk * fnn), moving ? vn : 1.0);
            if (moving) G = F - q;
        }
        if (__any_sync(0xffffffffu, contact && !moving)) {
            const double fp = F - fn;
            const double fpn = sqrt_alu(lane_sum(fp * fp, j));
            if (!moving && fs * fnn > fpn) G = F - fp;
        }
    }
    G = G + n * ((-disp) * kNormal);
    return contact ? G : F;
}

// What a lane keeps of its mass over a launch.
struct LaneMass {
    int64_t g;
    int c, j;
    bool on;           // the lane has a component of a free mass
    uint8_t fl;
    double m, gm;      // mass, and its weight's component g_c m
    AluDivisor md;     // the mass as a divisor (md_ok)
    bool md_ok;
    double x0, v0;     // RK2: the step's starting state
    double acc0;       // VERLET: the acceleration of the step before
};

// One step (RK2: half step) of the lane's component: F its summed spring
// force; x, v updated.  Called by whole warps.
template <int INTEG>
__device__ __forceinline__ void integrate_lanes(const StepArgs &a, const TileInfo &ti, const DevParams *prm, LaneMass &L,
                                                double F, double &x, double &v, int write_acc, int rk2_stage) {
    const int64_t np = a.npad;
    const int c = L.c, j = L.j;
    if (INTEG == INTEG_RK2 && rk2_stage == 0) {
        L.x0 = x;
        L.v0 = v;
    }
    F = F + L.gm;
    if (L.on && (L.fl & MF_EXT)) F = F + reinterpret_cast<const double *>(a.ext)[c * np + L.g];
    for (int q = 0; q < prm->nplanes; q++) {
        const double *p = prm->plane[q];
        F = plane_lanes(p[c], p[3], p[4], p[5], x, v, F, j, L.on);
    }
    for (int q = 0; q < prm->nballs; q++) {
        const double *b = prm->ball[q];
        const double d = x - b[c];
        const double dist = sqrt_alu(lane_sum(d * d, j));
        if (L.on && dist <= b[3]) F = F + div_wide(kNormal * d, dist);
    }
    if (__any_sync(0xffffffffu, L.on && (L.fl & MF_BODYPLANE))) {
        const double *p = a.body_plane + 6 * (int64_t)ti.body;
        F = plane_lanes(p[c], p[3], p[4], p[5], x, v, F, j, L.on && (L.fl & MF_BODYPLANE));
    }
    if (__any_sync(0xffffffffu, L.on && (L.fl & MF_LOCAL))) {
        double xx[3], vv[3], FF[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xx[k] = __shfl_sync(0xffffffffu, x, k * kLaneMasses + j);
            vv[k] = __shfl_sync(0xffffffffu, v, k * kLaneMasses + j);
            FF[k] = __shfl_sync(0xffffffffu, F, k * kLaneMasses + j);
        }
        if (L.on && (L.fl & MF_LOCAL)) {
            local_apply(a, L.g, xx, vv, FF);
            F = c == 0 ? FF[0] : (c == 1 ? FF[1] : FF[2]);
            v = c == 0 ? vv[0] : (c == 1 ? vv[1] : vv[2]);
        }
    }
    if (__any_sync(0xffffffffu, L.on && (L.fl & MF_DRAG))) {
        const double vn = sqrt_alu(lane_sum(v * v, j));
        if (L.on && (L.fl & MF_DRAG) && vn != 0.0) {
            const double k = (double)(-a.drag[L.g]) * (vn * vn);
            F = F + div_alu(v * k, vn);
        }
    }
    uint32_t bad = 0;
    double acc = alu_pack(alu_div(alu_unpack(F, bad), L.md));
    if (alu_bad(bad) || !L.md_ok) acc = div_wide(F, L.m);
    const double dt = prm->dt;
    if (INTEG == INTEG_VERLET) {
        v = v + (0.5 * (L.acc0 + acc)) * dt;
        x = x + (v * dt + (0.5 * acc) * prm->dt2);
        L.acc0 = acc;
    } else if (INTEG == INTEG_RK2) {
        if (rk2_stage == 0) {
            x = x + (0.5 * v) * dt;
            v = v + (0.5 * acc) * dt;
        } else {
            x = L.x0 + v * dt;
            v = L.v0 + acc * dt;
        }
    } else {
        v = v + acc * dt;
        x = x + v * dt;
    }
    if (write_acc && L.on) reinterpret_cast<double *>(a.acc)[c * np + L.g] = acc;
}

}  // namespace
}  // namespace tg
