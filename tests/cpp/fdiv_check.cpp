// Checks div_step (qsl_gb300/csrc/lean.cuh) against the host's IEEE division
// by sqrt(2) in binary32: every significand, at several exponents and both
// signs, and the operands at the ends of the range that it takes.
#include "lean.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>

int main()
{
    const float d = float(std::sqrt(2)), r = 1.0f / d;
    long fails = 0, taken = 0;
    auto check = [&](uint32_t bits) {
        float x;
        std::memcpy(&x, &bits, 4);
        if (!qslc::emu::div_step_takes(x)) return;
        taken++;
        volatile float want = x / d;
        const float w = want, got = qslc::emu::div_step(x, d, r);
        if (std::memcmp(&w, &got, 4) != 0 && fails++ < 10) std::printf("%a / %a = %a, got %a\n", x, d, w, got);
    };
    for (uint32_t m = 0; m < (1u << 23); m++) check((127u << 23) | m);
    for (uint32_t e : {27u, 28u, 100u, 126u, 128u, 253u, 254u})
        for (uint32_t m = 0; m < (1u << 23); m += 4099) {
            check((e << 23) | m);
            check(0x80000000u | (e << 23) | m);
        }
    for (uint32_t b : {0u, 0x80000000u, 1u, 0x007FFFFFu, 27u << 23, 0x7F7FFFFFu, 0xFF7FFFFFu, 0x7F800000u}) check(b);
    std::printf("taken %ld fails %ld\n", taken, fails);
    if (fails || qslc::emu::div_step_takes(1e-40f) || qslc::emu::div_step_takes(INFINITY) ||
        qslc::emu::div_step_takes(NAN))
        return 1;
    std::printf("fdiv ok\n");
    return 0;
}
