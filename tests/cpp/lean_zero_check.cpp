// Checks the products of qsl_gb300/csrc/lean.cuh that take zeros of either sign
// beside easy operands (LeanOpZ), and the constants of make_lean_gate, powers
// of two among them, against the host's IEEE arithmetic, bit for bit.
#include "lean.cuh"

#include <cmath>
#include <cstdio>
#include <random>

using namespace qslc::emu;

static std::mt19937_64 rng(11);
static long fails = 0, taken = 0;

static double operand(int ef)
{
    uint64_t m = rng() & MANT;
    if (rng() % 3 == 0) m &= ~((uint64_t(1) << (rng() % 32)) - 1);
    return dfrom((uint64_t(ef) << 52) | m | ((rng() & 1) ? SIGN : 0));
}

static void check(const char *what, double a, double b, double want, uint64_t got)
{
    taken++;
    if (got != dbits(want) && fails++ < 10) std::printf("%s: %a, %a: %a, got %a\n", what, a, b, want, dfrom(got));
}

static void product(double a, double c, const LeanK &k)
{
    volatile double want = a * c;
    if (is_zero(dbits(a)) || easy_product(dbits(a))) check("with zeros", a, c, want, lean_mul(lean_operand_z(dbits(a)), k));
    if (easy_product(dbits(a))) check("easy", a, c, want, lean_mul(lean_operand(dbits(a)), k));
}

int main()
{
    const int efs[] = {1, 64, 65, 66, 900, 1023, 2043, 2044, 2045, 2046};
    for (int i = 0; i < 2000; i++) {
        const int e = i < 260 ? -(i >> 2) : -int(rng() % 5);
        uint64_t m = i < 260 ? HIDDEN : (rng() & MANT) | HIDDEN;
        const double c = std::ldexp(double(m), e - 52) * ((i & 1) ? -1.0 : 1.0);
        const LeanK k = make_lean_gate(c);
        if (!k.usable) {
            if (m == HIDDEN || (m & 0xFFFFF)) fails++;
            continue;
        }
        if (m != HIDDEN && !make_lean(c).usable) fails++;
        if (lean_sign(k) != (std::signbit(c) ? 0x80000000u : 0u)) fails++;
        for (double z : {0.0, -0.0}) product(z, c, k);
        for (int j = 0; j < 500; j++) product(operand(efs[rng() % 10]), c, k);
        // ends of the significand
        for (uint64_t d = 0; d < 4; d++)
            for (int ef : efs) {
                product(dfrom((uint64_t(ef) << 52) | (MANT - d)), c, k);
                product(dfrom((uint64_t(ef) << 52) | (d + 1)), c, k);
            }
    }
    const double refused[] = {0.0, -0.0, 2.0, -4.0, std::ldexp(1.0, -65), 0.75, -1.5, 1e-320, INFINITY, NAN};
    for (double c : refused)
        if (make_lean_gate(c).usable) fails++;
    std::printf("taken %ld fails %ld\n", taken, fails);
    if (fails || taken < 1000000) return 1;
    std::printf("lean zero ok\n");
    return 0;
}
