// fp64_alu.cuh -- FP64 square root, division, product and sine on the integer
// units.  The first three are correctly rounded (round to nearest even): the
// bits of the IEEE operation, which is what the FP64 form's parity with the
// CPU oracle needs.
//
// Why: GB300 executes 1.6 FP64 operations per SM and clock (measured, any of
// add, multiply, fma, compare or conversion: a warp instruction takes 20
// cycles of the SM), against 23 32x32->64-bit multiply-adds, 60 logic
// operations or shifts and 118 additions.  A square root or a division is
// eight or more FP64 instructions (160 cycles a warp); below, a division by
// a divisor whose reciprocal is at hand is about 13 cycles and a product
// about 12, and they leave the FP64 pipe to the additions.  Measured, entry
// forces with square root, divisions and products here against all on the
// FP64 pipe, per step: 70^3 lattice 0.93 -> 0.48 ms, 96 bodies of 3-9 masses
// per side 87 -> 49 us, a 24x19x27 block with RK2 99 -> 55 us.
//
// Method: operands are split into a 53-bit integer significand and an
// exponent.  The square root and the quotient are integers Q with a known
// exact remainder condition: an estimate from a reciprocal (square root)
// good to about 2^-59 -- a 22-bit FP32 hardware estimate improved by one
// third-order step, y (1 + e/2 + 3 e^2/8) with e = 1 - n y^2, or y (1 - f +
// f^2) with f = n y - 1 (over all FP32 significands |e| < 2^-20.8 and
// |f| < 2^-21.8 on the GPU, so what the step leaves out is below 2^-64) -- gives Q to within a little more than half a unit,
// biased down, and the exact remainder modulo 2^64 (it is far smaller than
// 2^63 in magnitude) says whether the next integer is nearer.  Neither a
// quotient nor a square root of 53-bit operands can lie half-way between two
// 53-bit numbers, so no tie arises; a product's does, and is rounded from
// its exact 106 bits.
//
// Range: operands are zero or normal with exponents in [-255, 256].  alu_unpack
// collects in `bad` what is outside (subnormals, infinities, NaN, huge and
// tiny values); the caller then uses the FP64 instructions.  A zero carries
// an exponent far below any other through products and quotients.
//
// The host compiles the same functions, with its own initial estimates, for
// the test against IEEE results and the C library's sine
// (tests/test_fp64_alu_cpu.py).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define TG_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define TG_HD inline
#endif

namespace tg {

// value = (-1)^s m 2^(e - 1075), m in [2^52, 2^53) (functions say where 2^53
// may be returned and is taken).  se holds the sign in bit 31 and e + kAluBias
// below it, so that one addition gives a product's sign and exponent; e < 0,
// bit 20 clear, is a zero.
struct Alu {
    uint64_t m;
    uint32_t se;
};
constexpr uint32_t kAluBias = 0x100000u, kAluZeroDrop = 0x8000u;
// nonzero operands in range leave these bits of `bad` clear
constexpr uint32_t kAluBadBits = 0x60000000u;

TG_HD uint64_t alu_bits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
TG_HD double alu_double(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
TG_HD uint64_t alu_join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
TG_HD uint32_t alu_lo(uint64_t x) { return (uint32_t)x; }
TG_HD uint32_t alu_hi(uint64_t x) { return (uint32_t)(x >> 32); }
TG_HD uint64_t alu_mad(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }  // one IMAD.WIDE
TG_HD uint32_t alu_mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// the low 32 bits of (hi : lo) >> s, s < 32
TG_HD uint32_t alu_shr(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)(((((uint64_t)hi) << 32) | lo) >> s);
#endif
}
// the high 64 bits of a 64 x 64 product, at most 3 too small
TG_HD uint64_t alu_mulhi64(uint64_t a, uint64_t b) {
    return alu_mad(alu_hi(a), alu_hi(b), (uint64_t)alu_mulhi(alu_hi(a), alu_lo(b)) + alu_mulhi(alu_lo(a), alu_hi(b)));
}
// the low 64 bits of a 64 x 64 product
TG_HD uint64_t alu_mullo64(uint64_t a, uint64_t b) {
    const uint64_t p = (uint64_t)alu_lo(a) * alu_lo(b);
    return alu_join(alu_hi(p) + alu_lo(a) * alu_hi(b) + alu_hi(a) * alu_lo(b), alu_lo(p));
}
TG_HD uint32_t alu_float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
TG_HD float alu_float(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}
#ifndef __CUDA_ARCH__
// the host's estimates, moved by a number of units that a test chooses
#ifndef TG_ALU_HOST_SHIFT
#define TG_ALU_HOST_SHIFT 0
#endif
inline float alu_host_estimate(float y) { return alu_float(alu_float_bits(y) + (uint32_t)(TG_ALU_HOST_SHIFT)); }
#endif
// 1/sqrt(x), 1/x, good to 22 bits
TG_HD float alu_rsqrt_estimate(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return alu_host_estimate(1.0f / std::sqrt(x));
#endif
}
TG_HD float alu_rcp_estimate(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return alu_host_estimate(1.0f / x);
#endif
}

TG_HD Alu alu_unpack(double x, uint32_t &bad) {
    const uint64_t b = alu_bits(x);
    const uint32_t h = alu_hi(b);
    Alu a;
    a.m = alu_join((h & 0xfffffu) | 0x100000u, alu_lo(b));
    a.se = ((uint32_t)((int32_t)h >> 20) & 0x800007ffu) | kAluBias;
    if (((h & 0x7fffffffu) | alu_lo(b)) == 0)
        a.se -= kAluZeroDrop;
    else
        bad |= (h + 0x10000000u) ^ 0x40000000u;  // exponent fields 768..1279: bits 30, 29 = 1, 0
    return a;
}
TG_HD bool alu_bad(uint32_t bad) { return (bad & kAluBadBits) != 0; }
TG_HD bool alu_nonzero(const Alu &a) { return (a.se & kAluBias) != 0; }

// m may be 2^53
TG_HD double alu_pack(const Alu &a) {
    const uint32_t h = alu_hi(a.m) + (a.se << 20) - 0x100000u;  // m's top bit adds one to the exponent field
    const bool nz = alu_nonzero(a);
    return alu_double(alu_join(((nz ? h : 0u) & 0x7fffffffu) | (a.se & 0x80000000u), nz ? alu_lo(a.m) : 0u));
}

// m = 2^53 (a significand rounded up over the top) becomes 2^52
TG_HD void alu_carry(Alu &a) {
    const uint32_t c = alu_hi(a.m) >> 21;
    a.m = alu_join(alu_hi(a.m) >> c, alu_lo(a.m));  // the low bits of 2^53 are zero
    a.se += c;
}

// The 106-bit product hi : w (hi in [2^52, 2^54), w the 32 bits below it with
// a sticky lowest bit) rounded to 53 bits.
TG_HD Alu alu_round(uint64_t hi, uint32_t w, uint32_t se) {
    const uint32_t s = alu_hi(hi) >> 21;  // 1: hi has 54 bits
    uint32_t h = alu_hi(hi) >> s, l = alu_shr(alu_lo(hi), alu_hi(hi), s);
    // below the half-way bit: the sticky bit, and l's lowest (half-way cases
    // go to the even neighbour)
    w = alu_shr(w, alu_lo(hi), s) | ((w | l) & 1u);
#ifdef __CUDA_ARCH__
    // w above one half carries into the significand
    asm("add.cc.u32 %2, %2, 0x7fffffff;\n addc.cc.u32 %0, %0, 0;\n addc.u32 %1, %1, 0;" : "+r"(l), "+r"(h), "+r"(w));
    return Alu{alu_join(h, l), se + s};
#else
    return Alu{alu_join(h, l) + (w > 0x80000000u ? 1u : 0u), se + s};
#endif
}
TG_HD uint32_t alu_sticky(uint32_t x) { return x < 1u ? x : 1u; }

// a * b; a's m may be 2^53, and the result's
TG_HD Alu alu_mul(const Alu &a, const Alu &b) {
    const uint64_t x = a.m << 1, y = b.m << 11;
    const uint32_t xl = alu_lo(x), xh = alu_hi(x), yl = alu_lo(y), yh = alu_hi(y);
    const uint64_t p = alu_mad(xl, yl, 0);
    const uint64_t t = alu_mad(xl, yh, alu_hi(p));
    const uint64_t u = alu_mad(xh, yl, alu_lo(t));
    const uint64_t hi = alu_mad(xh, yh, (uint64_t)alu_hi(t)) + alu_hi(u);
    return alu_round(hi, alu_lo(u) | alu_sticky(alu_lo(p)), a.se + b.se - (1023u + kAluBias));
}

TG_HD Alu alu_square(const Alu &a) {
    const uint64_t x = a.m << 6;  // 59 bits: x^2 = m^2 2^12
    const uint32_t xl = alu_lo(x), xh = alu_hi(x);
    const uint64_t p = alu_mad(xl, xl, 0);
    const uint64_t t = alu_mad(xl, xh << 1, alu_hi(p));  // xh < 2^27
    const uint64_t hi = alu_mad(xh, xh, (uint64_t)alu_hi(t));
    return alu_round(hi, alu_lo(t) | alu_sticky(alu_lo(p)), a.se + a.se - (1023u + kAluBias));
}

// A divisor: significand, sign and exponent, and reciprocal r = 2^115 / m
// (2^62 <= r <= 2^63), relative error below 2^-58.5.
struct AluDivisor {
    uint64_t m, r;
    uint32_t se;
};

// a / d
TG_HD Alu alu_div(const Alu &a, const AluDivisor &d) {
    const bool lt = a.m < d.m;
    const uint64_t x = lt ? a.m << 1 : a.m;        // x / d.m in [1, 2)
    const uint64_t t = alu_mulhi64(x << 10, d.r);  // (x / d.m) 2^61, within 24
    // nearest integer from below: 64 units of 2^-9 short of half
    uint64_t q = (t + (256u - 64u)) >> 9;
    // exact remainder x 2^52 - q d.m
    const uint64_t rem = alu_join(alu_lo(x) << 20, 0) - alu_mullo64(q, d.m);
    q += alu_hi(d.m - (rem << 1)) >> 31;
    return Alu{q, a.se - d.se + (1023u + kAluBias) - (lt ? 1u : 0u)};
}

// |x| as a divisor from its unpacked form (not zero)
TG_HD AluDivisor alu_divisor(const Alu &x) {
    // y23 2^-23 = 1/v, v = m 2^-52 in [1, 2)
    const float v = alu_float(0x3f800000u | alu_lo(x.m >> 29));  // m's bit 52 lands on exponent bit 0, set already
    const uint32_t y = alu_float_bits(alu_rcp_estimate(v) + 1.0f) - 0x3f800000u;
    // f = v y - 1: m y in units of 2^-75 -> keep 2^-64 (modulo 1: |f| < 2^-21)
    const uint64_t lo = (uint64_t)alu_lo(x.m) * y;
    const uint64_t prod_hi = alu_mad(alu_hi(x.m), y, lo >> 32);  // units of 2^-43
    const uint64_t f64 = (prod_hi << 21) | (alu_lo(lo) >> 11);
    const int32_t ft = (int32_t)((int64_t)f64 >> 16);            // units of 2^-48
    const uint32_t ft_abs = (uint32_t)(ft < 0 ? -ft : ft);
    const uint64_t c = f64 - alu_mulhi(ft_abs, ft_abs);          // f - f^2, units of 2^-64
    // r = 2^63 y23 2^-23 (1 - c)
    const uint64_t yc = ((uint64_t)y * alu_lo(c)) >> 24;         // 2^63 2^-23 2^-64 = 2^-24
    const int64_t yh = (int64_t)(int32_t)alu_hi(c) * (int32_t)y; // times 2^32: << 8
    return AluDivisor{x.m, ((uint64_t)y << 40) - (uint64_t)(yh * 256) - yc, x.se};
}

// sqrt of the positive number n, and the result as a divisor
TG_HD Alu alu_sqrt(const Alu &n, AluDivisor &d) {
    // n = N 2^(2h), N in [2^52, 2^54)
    const uint32_t odd = (n.se & 1u) ^ 1u;  // of e - 1075
    const uint64_t N = odd ? n.m << 1 : n.m;
    // y 2^-23 = 1/sqrt(N 2^-52)
    const float v = alu_float((0x3f800000u + (odd << 23)) | (alu_lo(n.m >> 29) & 0x7fffffu));
    const uint32_t y = alu_float_bits(alu_rsqrt_estimate(v) + 1.0f) - 0x3f800000u;
    // e = 1 - N y^2, in units of 2^-66 modulo 2^64 (|e| < 2^-19)
    const uint64_t P = (uint64_t)y * y;
    uint64_t t = alu_mad(alu_hi(N), alu_lo(P), alu_mulhi(alu_lo(N), alu_lo(P)));
    t = alu_mad(alu_lo(N), alu_hi(P), t);
    t += (uint64_t)(alu_hi(N) * alu_hi(P)) << 32;
    const int64_t e = (int64_t)(0 - t);
    const int32_t et = (int32_t)(e >> 16);                       // units of 2^-50
    const uint32_t et_abs = (uint32_t)(et < 0 ? -et : et);
    const uint32_t e2 = alu_mulhi(et_abs, et_abs);               // e^2, units of 2^-68
    const int64_t c = (e >> 1) + ((e2 * 3u) >> 5);               // e/2 + 3 e^2/8, 2^-66
    // y63 = 2^63 y 2^-23 (1 + c)
    const uint64_t cl = ((uint64_t)y * alu_lo((uint64_t)c)) >> 26;
    const int64_t ch = (int64_t)(int32_t)alu_hi((uint64_t)c) * (int32_t)y;  // times 2^32: << 6
    const uint64_t y63 = ((uint64_t)y << 40) + (uint64_t)(ch * 64) + cl;
    // S = sqrt(N 2^52) from below, then the exact remainder N 2^52 - S^2
    const uint64_t sx = alu_mulhi64(N << 10, y63);               // sqrt(N 2^-52) 2^61
    uint64_t S = (sx + (256u - 64u)) >> 9;
    const uint64_t p = (uint64_t)alu_lo(S) * alu_lo(S);
    const uint64_t sq = alu_join(alu_hi(p) + alu_lo(S) * (alu_hi(S) << 1), alu_lo(p));
    uint64_t rho = alu_join(alu_lo(N) << 20, 0) - sq;
    const uint32_t up = alu_hi(S - rho) >> 31;                   // rho > S: S + 1 is nearer
    rho -= up ? ((S << 1) | 1u) : 0;
    S += up;
    // 1/S = 1/sqrt(N 2^52) (1 + rho / (2 S^2)): rho y^3 2^-42 in y63's units
    const uint32_t y16 = alu_hi(y63) >> 15;
    const uint32_t y3 = (((y16 * y16) >> 16) * y16) >> 16;  // y16 = 2^16 where y = 1
    const int32_t corr = ((int32_t)alu_hi(rho) * (int32_t)(y3 >> 7)) >> 19;
    // e of the root: (e - 1075 - odd) / 2 - 26 + 1075
    const uint32_t se = ((n.se - kAluBias + 1023u - odd) >> 1) + kAluBias;
    d = AluDivisor{S, y63 + (uint64_t)(int64_t)corr, se};
    return Alu{S, se};
}

// sin(x) for 2^-24 <= |x| < 2^30 (alu_sin_range): the turn fraction x / 2 pi
// modulo 1 from the exact product of the significand with 96 bits of 1/2 pi,
// folded to a quarter turn X and summed as X (d0 - t (d1 - t (d2 - ...))),
// t = X^2, d_k = (pi/2)^(2k+1) / (2k+1)!: the Taylor series of the sine, cut
// where its terms are below 2^-67.  Absolute error below 2^-59 before the
// one rounding to 53 bits.
TG_HD bool alu_sin_range(double x) {
    const uint32_t e = (alu_hi(alu_bits(x)) >> 20) & 0x7ffu;
    return e - (1023u - 24u) < 54u;
}

TG_HD Alu alu_sin(double x) {
    const uint64_t b = alu_bits(x);
    const uint32_t bh = alu_hi(b);
    const uint32_t mh = (bh & 0xfffffu) | 0x100000u, ml = alu_lo(b);
    const uint32_t e = (bh >> 20) & 0x7ffu;
    // |x| / 2 pi = (m K) 2^(e - 1075 - 96); words w4..w1 of m K (w0 dropped)
    constexpr uint32_t k2 = 0x28be60dbu, k1 = 0x9391054au, k0 = 0x7f09d5f4u;
    uint64_t lo = alu_mad(ml, k1, alu_mulhi(ml, k0));
    const uint64_t hi = alu_mad(ml, k2, alu_hi(lo));
    uint64_t r = alu_mad(mh, k0, alu_lo(lo));
    const uint32_t w1 = alu_lo(r);
    r = alu_mad(mh, k1, (uint64_t)alu_lo(hi) + alu_hi(r));
    const uint32_t w2 = alu_lo(r);
    r = alu_mad(mh, k2, (uint64_t)alu_hi(hi) + alu_hi(r));
    const uint32_t w3 = alu_lo(r), w4 = alu_hi(r);
    // the 64 bits below the binary point: bit 1107 - e - 32 (of w1's lowest
    // upwards) in [23, 76]
    const uint32_t at = 1075u - e;
    const uint32_t v0 = at >= 64 ? w3 : (at >= 32 ? w2 : w1), v1 = at >= 64 ? w4 : (at >= 32 ? w3 : w2),
                   v2 = at >= 64 ? 0u : (at >= 32 ? w4 : w3);
    uint32_t f0 = alu_shr(v0, v1, at & 31), f1 = alu_shr(v1, v2, at & 31);
    // fold: turns in [1/4, 3/4) are mirrored; then |turns| <= 1/4
    const bool mirror = ((f1 + 0x40000000u) & 0x80000000u) != 0;
    uint64_t f = alu_join(f1, f0);
    if (mirror) f = 0x8000000000000000ull - f;
    const uint32_t neg = alu_hi(f) & 0x80000000u;
    if (neg) f = 0 - f;
    // X and t in units of 2^-64, the terms from k = 6 down in 2^-63
    const uint64_t X = f >= 0x4000000000000000ull ? ~0ull : f << 2;
    const uint64_t T = alu_mulhi64(X, X);
    const uint32_t t = alu_hi(T);
    uint32_t q = 0x251u - alu_mulhi(t, 3u);  // units of 2^-61, from k = 10
    q = 0x18a40u - alu_mulhi(t, q);
    q = 0xd57619u - alu_mulhi(t, q);
    q = 0x5beb6e7cu - alu_mulhi(t, q);
    uint64_t p = 0x7a3d0d3406ull - ((uint64_t)alu_mulhi(t, q) << 2);
    p = 0x1e3074fde887ull - alu_mulhi64(T, p);
    p = 0x541e0d21fb9e0ull - alu_mulhi64(T, p);
    p = 0x9969667315ec2eull - alu_mulhi64(T, p);
    p = 0xa335e33bad570e9ull - alu_mulhi64(T, p);
    p = 0x52aef39896f94afbull - alu_mulhi64(T, p);
    p = 0xc90fdaa22168c235ull - alu_mulhi64(T, p);
    uint64_t s = alu_mulhi64(X, p);
    // to 53 bits, round to nearest
    Alu a;
#ifdef __CUDA_ARCH__
    const int z = __clzll((long long)s);
#else
    const int z = s ? __builtin_clzll(s) : 64;
#endif
    s <<= z & 63;
    a.m = (s + 0x400u) >> 11;
    if (s > ~0ull - 0x400u) a.m = 1ull << 53;
    a.se = ((bh & 0x80000000u) ^ neg) | (kAluBias + (s ? 1023u - (uint32_t)z : 0u - kAluZeroDrop));
    return a;
}

}  // namespace tg
