// Checks the products and the division of qsl_gb300/csrc/lean.cuh against
// the host's IEEE arithmetic, bit for bit, over the operands that they
// accept: random significands, few-bit ones, ones whose product or quotient
// sits next to the threshold that chooses the shift, next to a rounding
// carry, and next to a rounding midpoint, at both ends of the exponent range.
#include "lean.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace qslc::emu;
typedef unsigned __int128 u128;

static std::mt19937_64 rng(7);

static uint64_t significand()
{
    uint64_t m = rng() & MANT;
    switch (rng() % 4) {
    case 0: m &= ~((uint64_t(1) << (rng() % 32)) - 1); break;
    case 1: m = (rng() % 64) << (rng() % 46); break;
    default: break;
    }
    return (m & MANT) | HIDDEN;
}

static double build(uint64_t m, int ef, bool neg)
{
    return dfrom((uint64_t(ef) << 52) | (m & MANT) | (neg ? SIGN : 0));
}

static long fails = 0, taken = 0, refused = 0, unsure = 0;

static void product(uint64_t ma, int ef, double c, const LeanK &k)
{
    const double a = build(ma, ef, rng() & 1);
    if (!easy_product(dbits(a))) {
        refused++;
        return;
    }
    volatile double want = a * c;
    const uint64_t got = lean_mul(lean_operand(dbits(a)), k);
    taken++;
    if (got != dbits(want) && fails++ < 10)
        std::printf("product: %a * %a = %a, got %a\n", a, c, double(want), dfrom(got));
}

static void quotient(uint64_t mx, int ef, double y, const LeanDiv &k)
{
    const double x = build(mx, ef, rng() & 1);
    if (!easy_range(dbits(x))) {
        refused++;
        return;
    }
    bool sure = true;
    const uint64_t got = lean_div(lean_operand(dbits(x)), k, sure);
    if (!sure) {
        unsure++;
        return;
    }
    volatile double want = x / y;
    taken++;
    if (got != dbits(want) && fails++ < 10)
        std::printf("quotient: %a / %a = %a, got %a\n", x, y, double(want), dfrom(got));
}

int main(int argc, char **argv)
{
    const long count = argc > 1 ? std::atol(argv[1]) : 1000000;
    const int efs[] = {0, 1, 64, 65, 66, 900, 1022, 1023, 1024, 2043, 2044, 2045, 2046, 2047};
    // products
    for (int ci = 0; ci < 400; ci++) {
        const int e = ci % 5 == 0 ? -int(rng() % 65) : -int(rng() % 3);
        uint64_t mc = significand();
        const double c = std::ldexp(double(mc), e - 52) * ((rng() & 1) ? -1.0 : 1.0);
        const LeanK k = make_lean(c);
        if (!k.usable) {
            refused++;
            continue;
        }
        for (long i = 0; i < count / 400; i++) product(significand(), efs[rng() % 14], c, k);
        const uint64_t t = uint64_t(((u128(1) << 105) + mc - 1) / mc);        // the shift's threshold
        for (int d = -3; d <= 3; d++)
            for (int ef : efs) {
                const uint64_t m = t + uint64_t(int64_t(d));
                if (m >= HIDDEN && m < 2 * HIDDEN) product(m, ef, c, k);
            }
        // near-midpoint products: ma * mc = half + small mod 2^52 (or 2^53)
        for (int top = 0; top < 2; top++) {
            const uint64_t mod = uint64_t(1) << (52 + top), odd = mc | 1;
            uint64_t inv = odd;                                             // inverse of odd mod 2^64
            for (int it = 0; it < 6; it++) inv *= 2 - odd * inv;
            for (int64_t off = -4; off <= 4; off++) {
                const uint64_t ma = ((mod / 2 + uint64_t(off)) * inv) & (mod - 1);
                const double co = std::ldexp(double(odd), e - 52);
                const LeanK ko = make_lean(co);
                for (uint64_t add = 0; add < 4; add++) {
                    const uint64_t m = ma + add * mod;
                    if (ko.usable && m >= HIDDEN && m < 2 * HIDDEN) product(m, 1022, co, ko);
                }
            }
            // products that round up to the next power of two
            const u128 hi = u128(1) << (105 + top);
            const uint64_t m = uint64_t((hi - 1) / mc);
            for (uint64_t d = 0; d < 3; d++)
                if (m - d >= HIDDEN && m - d < 2 * HIDDEN)
                    for (int ef : efs) product(m - d, ef, c, k);
        }
    }
    // constants the products must refuse: more than 19 trailing zeros
    if (make_lean(1.0).usable || make_lean(0.5).usable || make_lean(0.0).usable || make_lean(2.0).usable ||
        make_lean(std::ldexp(double((uint64_t(1) << 32) + 1), -32)).usable)
        fails++;
    // quotients by sqrt(2) and by random divisors
    for (int yi = 0; yi < 50; yi++) {
        const double y = yi == 0 ? std::sqrt(2.0) : std::ldexp(double(significand()), int(rng() % 3) - 53);
        const LeanDiv k = make_lean_div(y);
        if (!k.usable) {
            refused++;
            if (yi == 0) fails++;
            continue;
        }
        const uint64_t my = (dbits(y) & MANT) | HIDDEN;
        for (long i = 0; i < count / 50; i++) quotient(significand(), efs[rng() % 14], y, k);
        for (int64_t d = -3; d <= 3; d++)
            for (int ef : efs) {
                const uint64_t m = my + uint64_t(d);
                if (m >= HIDDEN && m < 2 * HIDDEN) quotient(m, ef, y, k);
            }
        // quotients next to a midpoint and next to an integer:
        // mx * 2^k53 = (t + 1/2) * my or t * my, off by a little
        for (int i = 0; i < 2000; i++) {
            const int sh = int(rng() & 1);
            const u128 t = (u128(1) << 52) + (rng() & MANT);
            for (int half = 0; half < 2; half++) {
                const uint64_t m = uint64_t(((2 * t + unsigned(half)) * my) >> (53 + sh));
                for (int64_t d = -1; d <= 1; d++) {
                    const uint64_t x = m + uint64_t(d);
                    if (x >= HIDDEN && x < 2 * HIDDEN) quotient(x, 1023, y, k);
                }
            }
        }
    }
    std::printf("taken %ld refused %ld unsure %ld fails %ld\n", taken, refused, unsure, fails);
    // a divisor's undecided quotients are a few in 2^29 of random ones
    if (unsure * 1000 > taken) fails++;
    if (fails) return 1;
    std::printf("lean ok\n");
    return 0;
}
