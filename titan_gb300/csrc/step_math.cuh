// step_math.cuh -- device-side force functions of the step kernels: the
// reference constraint forces in FP64 (reference operation order) and FP32,
// and error-free float transformations for the compensated update.
#pragma once

#include "engine.h"
#include "fp64_alu.cuh"

namespace tg {
namespace {

constexpr double kNormal = 20000.0;  // src/object.cu:26

// ---------------------------------------------------------------- FP64 ----
__device__ __forceinline__ double nrm3(double a, double b, double c) {
    return sqrt((a * a + b * b) + c * c);
}
__device__ __forceinline__ double dot3(const double *a, const double *b) {
    return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}

// The same with the products and the square root on the integer units
// (fp64_alu.cuh: the same bits), and a vector times or divided by a number;
// the _wide forms serve operands outside the integer path's range and are
// kept out of line.  The epilogue then has 19 FP64 instructions per mass
// where it had about 92 (a plane, a ball, Euler).
struct D3 {
    double x, y, z;
};
__device__ __noinline__ double dot3_wide(double a0, double a1, double a2, double b0, double b1, double b2) {
    return (a0 * b0 + a1 * b1) + a2 * b2;
}
__device__ __noinline__ double nrm3_wide(double a, double b, double c) { return nrm3(a, b, c); }
__device__ __noinline__ D3 mul3_wide(double a0, double a1, double a2, double b) { return D3{a0 * b, a1 * b, a2 * b}; }
__device__ __noinline__ D3 div3_wide(double a0, double a1, double a2, double b) { return D3{a0 / b, a1 / b, a2 / b}; }

__device__ __forceinline__ double dot3_alu(const double *a, const double *b) {
    uint32_t bad = 0;
    double p[3];
#pragma unroll
    for (int c = 0; c < 3; c++) p[c] = alu_pack(alu_mul(alu_unpack(a[c], bad), alu_unpack(b[c], bad)));
    if (alu_bad(bad)) return dot3_wide(a[0], a[1], a[2], b[0], b[1], b[2]);
    return (p[0] + p[1]) + p[2];
}
__device__ __forceinline__ double nrm3_alu(double a, double b, double c) {
    uint32_t bad = 0;
    const double q0 = alu_pack(alu_square(alu_unpack(a, bad))), q1 = alu_pack(alu_square(alu_unpack(b, bad))),
                 q2 = alu_pack(alu_square(alu_unpack(c, bad)));
    const Alu n2 = alu_unpack((q0 + q1) + q2, bad);
    if (alu_bad(bad) || !alu_nonzero(n2)) return nrm3_wide(a, b, c);
    AluDivisor d;
    return alu_pack(alu_sqrt(n2, d));
}
__device__ __forceinline__ D3 mul3_alu(const double *a, double b) {
    uint32_t bad = 0;
    const Alu y = alu_unpack(b, bad);
    const D3 r = {alu_pack(alu_mul(alu_unpack(a[0], bad), y)), alu_pack(alu_mul(alu_unpack(a[1], bad), y)),
                  alu_pack(alu_mul(alu_unpack(a[2], bad), y))};
    return alu_bad(bad) ? mul3_wide(a[0], a[1], a[2], b) : r;
}
__device__ __forceinline__ D3 div3_alu(const double *a, double b) {
    uint32_t bad = 0;
    const Alu y = alu_unpack(b, bad);
    const AluDivisor d = alu_divisor(y);
    const D3 r = {alu_pack(alu_div(alu_unpack(a[0], bad), d)), alu_pack(alu_div(alu_unpack(a[1], bad), d)),
                  alu_pack(alu_div(alu_unpack(a[2], bad), d))};
    return alu_bad(bad) || !alu_nonzero(y) ? div3_wide(a[0], a[1], a[2], b) : r;
}

// The force on a mass below a plane, from the force F so far.  Out of line:
// most warps have no mass in contact.
__device__ __noinline__ D3 plane_contact(double n0, double n1, double n2, double disp, double fk, double fs, double v0,
                                         double v1, double v2, double F0, double F1, double F2) {
    const double n[3] = {n0, n1, n2}, v[3] = {v0, v1, v2};
    double F[3] = {F0, F1, F2};
    const D3 fn3 = mul3_alu(n, dot3_alu(F, n));
    if (fs > 0 || fk > 0) {
        const D3 nv = mul3_alu(n, dot3_alu(v, n));
        const double vp[3] = {v[0] - nv.x, v[1] - nv.y, v[2] - nv.z};
        const double vn = nrm3_alu(vp[0], vp[1], vp[2]);
        if (vn > 1e-16) {
            const D3 t = mul3_alu(vp, fk * nrm3_alu(fn3.x, fn3.y, fn3.z));
            const double tv[3] = {t.x, t.y, t.z};
            const D3 q = div3_alu(tv, vn);
            F[0] = F[0] - q.x;
            F[1] = F[1] - q.y;
            F[2] = F[2] - q.z;
        } else {
            const double fp[3] = {F[0] - fn3.x, F[1] - fn3.y, F[2] - fn3.z};
            if (fs * nrm3_alu(fn3.x, fn3.y, fn3.z) > nrm3_alu(fp[0], fp[1], fp[2])) {
                F[0] = F[0] - fp[0];
                F[1] = F[1] - fp[1];
                F[2] = F[2] - fp[2];
            }
        }
    }
    const D3 q = mul3_alu(n, (-disp) * kNormal);
    return D3{F[0] + q.x, F[1] + q.y, F[2] + q.z};
}

// src/object.cu:73-106
__device__ __forceinline__ void plane_apply(const double *n, double off, double fk, double fs,
                                            const double *x, const double *v, double *F) {
    double disp = dot3_alu(x, n) - off;
    if (!(disp < 0)) return;  // only zeros would be added otherwise
    const D3 r = plane_contact(n[0], n[1], n[2], disp, fk, fs, v[0], v[1], v[2], F[0], F[1], F[2]);
    F[0] = r.x;
    F[1] = r.y;
    F[2] = r.z;
}

// F with the drag of a mass at velocity v added (src/sim.cu:1134-1137).
__device__ __noinline__ D3 drag_added(double v0, double v1, double v2, int32_t drag, double F0, double F1, double F2) {
    const double v[3] = {v0, v1, v2};
    const double vn = nrm3_alu(v0, v1, v2);
    if (!(vn != 0.0)) return D3{F0, F1, F2};
    const D3 t = mul3_alu(v, (double)(-drag) * (vn * vn));
    const double tv[3] = {t.x, t.y, t.z};
    const D3 q = div3_alu(tv, vn);
    return D3{F0 + q.x, F1 + q.y, F2 + q.z};
}

// src/object.cu:53-56
__device__ __forceinline__ void ball_apply(const double *c, double r, const double *x, double *F) {
    double d[3] = {x[0] - c[0], x[1] - c[1], x[2] - c[2]};
    double dist = nrm3_alu(d[0], d[1], d[2]);
    if (dist <= r) {
        F[0] = F[0] + (kNormal * d[0]) / dist;
        F[1] = F[1] + (kNormal * d[1]) / dist;
        F[2] = F[2] + (kNormal * d[2]) / dist;
    }
}

// src/object.cu:115-124
__device__ __forceinline__ void cplane_apply(const double *n, double fr, double *v, double *F) {
    double nf = dot3(F, n);
    F[0] = F[0] + (-n[0]) * nf;
    F[1] = F[1] + (-n[1]) * nf;
    F[2] = F[2] + (-n[2]) * nf;
    double vn = nrm3(v[0], v[1], v[2]);
    if (vn >= 1e-16) {
        double vdn = dot3(v, n);
        v[0] = v[0] + (-n[0]) * vdn;
        v[1] = v[1] + (-n[1]) * vdn;
        v[2] = v[2] + (-n[2]) * vdn;
        double s = (-fr) * nf;
        F[0] = F[0] + (v[0] * s) / vn;
        F[1] = F[1] + (v[1] * s) / vn;
        F[2] = F[2] + (v[2] * s) / vn;
    }
}

// src/object.cu:133-141
__device__ __forceinline__ void direction_apply(const double *t, double fr, double *v, double *F) {
    double fdt = dot3(F, t);
    double nf[3] = {F[0] - t[0] * fdt, F[1] - t[1] * fdt, F[2] - t[2] * fdt};
    F[0] = F[0] + (-nf[0]);
    F[1] = F[1] + (-nf[1]);
    F[2] = F[2] + (-nf[2]);
    if (nrm3(v[0], v[1], v[2]) >= 1e-16) {
        double vdt = dot3(v, t);
        v[0] = t[0] * vdt;
        v[1] = t[1] * vdt;
        v[2] = t[2] * vdt;
        double s = (-nrm3(nf[0], nf[1], nf[2])) * fr;
        F[0] = F[0] + t[0] * s;
        F[1] = F[1] + t[1] * s;
        F[2] = F[2] + t[2] * s;
    }
}

// Local constraints of one mass (src/sim.cu:1117-1131), records pre-sorted.
__device__ __forceinline__ void local_apply(const StepArgs &a, int64_t g, double *x, double *v,
                                            double *F) {
    for (int32_t r = a.lc_ptr[g]; r < a.lc_ptr[g + 1]; r++) {
        const double *rec = a.lc_rec + 4 * (int64_t)r;
        switch (a.lc_type[r]) {
            case 1: plane_apply(rec, rec[3], 0.0, 0.0, x, v, F); break;
            case 2: ball_apply(rec, rec[3], x, F); break;
            case 0: cplane_apply(rec, rec[3], v, F); break;
            case 3: direction_apply(rec, rec[3], v, F); break;
            default: break;
        }
    }
}

// ---------------------------------------------------------------- FP32 ----
__device__ __forceinline__ float nrm3f(float a, float b, float c) {
    return __fsqrt_rn(fmaf(c, c, fmaf(b, b, a * a)));
}
__device__ __forceinline__ float dot3f(const float *a, const float *b) {
    return fmaf(a[2], b[2], fmaf(a[1], b[1], a[0] * b[0]));
}

__device__ __forceinline__ void plane_applyf(const float *n, float disp, float fk, float fs,
                                             const float *v, float *F) {
    if (!(disp < 0.f)) return;
    float fdn = dot3f(F, n);
    float fn[3] = {n[0] * fdn, n[1] * fdn, n[2] * fdn};
    if (fs > 0.f || fk > 0.f) {
        float vdn = dot3f(v, n);
        float vp[3] = {v[0] - n[0] * vdn, v[1] - n[1] * vdn, v[2] - n[2] * vdn};
        float vn = nrm3f(vp[0], vp[1], vp[2]);
        if (vn > 1e-16f) {
            float fm = __fdiv_rn(fk * nrm3f(fn[0], fn[1], fn[2]), vn);
            F[0] -= vp[0] * fm;
            F[1] -= vp[1] * fm;
            F[2] -= vp[2] * fm;
        } else {
            float fp[3] = {F[0] - fn[0], F[1] - fn[1], F[2] - fn[2]};
            if (fs * nrm3f(fn[0], fn[1], fn[2]) > nrm3f(fp[0], fp[1], fp[2])) {
                F[0] -= fp[0];
                F[1] -= fp[1];
                F[2] -= fp[2];
            }
        }
    }
    float s = (-disp) * 20000.0f;
    F[0] += n[0] * s;
    F[1] += n[1] * s;
    F[2] += n[2] * s;
}

__device__ __forceinline__ void ball_applyf(const float *d, float r, float *F) {
    float dist = nrm3f(d[0], d[1], d[2]);
    if (dist <= r) {
        float s = __fdiv_rn(20000.0f, dist);
        F[0] += d[0] * s;
        F[1] += d[1] * s;
        F[2] += d[2] * s;
    }
}

// error-free transformations (Knuth two-sum, Dekker fast-two-sum)
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    e = __fsub_rn(b, __fsub_rn(s, a));
}

// 32-byte record as two read-only 16-byte loads
struct D4 { double x, y, z, w; };
__device__ __forceinline__ D4 ldg_d4(const double *p) {
    double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    return D4{a.x, a.y, b.x, b.y};
}

template <int PREC>
struct Real { using T = float; };
template <>
struct Real<P_FP64> { using T = double; };


}  // namespace
}  // namespace tg
