// Checks the square of qsl_gb300/csrc/lean.cuh against the host's IEEE multiply,
// bit for bit: random and few-bit significands, ones next to sqrt(2) (where the
// shift changes) and to a rounding carry, over the exponent fields that it
// accepts and at both ends; and that it refuses what lies outside.
#include "lean.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

using namespace qslc::emu;

static std::mt19937_64 rng(11);

int main(int argc, char **argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    const uint64_t root = 6369051672525772ull;          // floor(2^52.5)
    long fails = 0, taken = 0;
    for (long i = 0; i < n; i++) {
        uint64_t m = rng() & MANT;
        switch (rng() % 5) {
        case 0: m &= ~((uint64_t(1) << (rng() % 32)) - 1); break;
        case 1: m = (rng() % 64) << (rng() % 46); break;
        case 2: m = (root - 40 + rng() % 80) & MANT; break;
        case 3: m = rng() & 1 ? MANT - rng() % 64 : rng() % 64; break;
        default: break;
        }
        const int ends[6] = {511, 512, 513, 1532, 1533, 1534};
        const int ef = rng() % 3 ? 512 + int(rng() % 1022) : ends[rng() % 6];
        const uint64_t a = (uint64_t(ef) << 52) | m | (rng() & 1 ? SIGN : 0);
        const bool in = ef >= 512 && ef <= 1533 && (m & 0x1FFFFFF) != 0;
        if (easy_square(a) != in) fails++;
        if (!in) continue;
        taken++;
        const double x = dfrom(a);
        if (lean_square(a) != dbits(x * x)) fails++;
    }
    for (uint64_t a : {uint64_t(0), SIGN, uint64_t(1), uint64_t(0x7FF) << 52, (uint64_t(0x7FF) << 52) | 1})
        if (easy_square(a)) fails++;
    if (fails || taken < n / 4) {
        std::printf("%ld failures, %ld taken\n", fails, taken);
        return 1;
    }
    std::printf("square ok, %ld taken\n", taken);
}
