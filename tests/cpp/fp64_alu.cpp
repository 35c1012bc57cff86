// Host build of fp64_alu.cuh against the IEEE operations and the C library's
// sine.  Prints one line per check: name, operand sets, mismatches.  The
// reciprocal estimates are shifted by -3 to +3 units, because the GPU's
// differ from the host's by as much.
static int estimate_shift = 0;
#define TG_ALU_HOST_SHIFT estimate_shift
#include "fp64_alu.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>

using namespace tg;

static uint64_t seed = 0x9e3779b97f4a7c15ull;
static uint64_t rnd() {  // splitmix64 (Steele, Lea, Flood 2014)
    uint64_t z = (seed += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
// exponent in [lo, hi]; full, short, near-one-half-unit and all-ones significands
static double value(int lo, int hi, double zeros = 0.02) {
    uint64_t f = rnd() >> 12;
    const uint64_t cut = (1ull << (rnd() % 52)) - 1;
    switch (rnd() & 3) {
        case 1: f &= ~cut; break;
        case 2: f |= cut; break;
        case 3: f = ((1ull << 52) - 1) - (f & 7); break;
    }
    if ((double)(rnd() >> 11) * 0x1p-53 < zeros) return rnd() & 1 ? 0.0 : -0.0;
    return alu_double((rnd() & 1ull << 63) | (uint64_t)(lo + 1023 + (int)(rnd() % (uint64_t)(hi - lo + 1))) << 52 | f);
}
static bool same(double a, double b) { return alu_bits(a) == alu_bits(b); }

int main(int argc, char **argv) {
    const long sets = argc > 1 ? std::atol(argv[1]) : 1000000;
    long bad[5] = {0, 0, 0, 0, 0}, refused = 0, sines = 0;
    for (long i = 0; i < sets; i++) {
        estimate_shift = (int)(i % 7) - 3;
        const bool wide = (i & 1) != 0;
        const double a = wide ? value(-255, 256) : value(-8, 8), b = wide ? value(-255, 256) : value(-8, 8);
        uint32_t out = 0;
        const Alu x = alu_unpack(a, out), y = alu_unpack(b, out);
        refused += alu_bad(out);
        bad[0] += !same(alu_pack(alu_mul(x, y)), a * b);
        bad[1] += !same(alu_pack(alu_square(x)), a * a);
        if (alu_nonzero(y)) bad[2] += !same(alu_pack(alu_div(x, alu_divisor(y))), a / b);
        if (alu_nonzero(y)) {  // the root, and a quotient by it
            AluDivisor d;
            uint32_t o = 0;
            const double n = std::fabs(b), r = alu_pack(alu_sqrt(alu_unpack(n, o), d));
            bad[3] += !same(r, std::sqrt(n));
            bad[3] += !same(alu_pack(alu_div(x, d)), a / std::sqrt(n));
        }
        const double th = value(-24, 29, 0.0);
        if (alu_sin_range(th)) {
            sines++;
            // half a unit of the result, and the method's 2^-59
            const long double want = sinl((long double)th);
            const double got = alu_pack(alu_sin(th));
            const long double unit = std::ldexp(1.0L, want == 0 ? -1074 : std::ilogb((double)want) - 52);
            bad[4] += !(fabsl((long double)got - want) <= 0.5L * unit + 0x1p-59L);
        }
    }
    // operands that have to be refused: subnormal, infinite, NaN, outside [-255, 256]
    const double out_of_range[] = {5e-324, 2.2e-308, INFINITY, -INFINITY, NAN, 0x1p-256, 0x1p257, -0x1p1023};
    long taken = 0;
    for (double v : out_of_range) {
        uint32_t o = 0;
        (void)alu_unpack(v, o);
        taken += !alu_bad(o);
    }
    const char *name[] = {"product", "square", "quotient", "root", "sine"};
    for (int q = 0; q < 5; q++) std::printf("%s %ld %ld\n", name[q], q == 4 ? sines : sets, bad[q]);
    std::printf("refused %ld %ld\ntaken %d %ld\n", sets, refused, (int)(sizeof(out_of_range) / 8), taken);
    return 0;
}
