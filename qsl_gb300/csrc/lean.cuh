// lean.cuh -- exact binary64 products and a division by a constant on the
// integer pipes, for operands that need no special cases.
//
// dpemu.cuh's prod_pack takes any operand: it tests each one for zero and
// for its range, and shifts every product into place after multiplying.
// The forms here take only "easy" operands -- normal, exponent field 65 to
// 2044, low significand word not zero -- and leave every other operand to
// the caller, which tests them first (easy_range, easy_product) and sends a
// thread through the general path when it has one that is not easy.  What the
// restriction buys:
//   - no zero handling (LeanOpZ adds it, for the threads that need it), and
//     no rounding ties: a product lies half-way
//     between two doubles only when the operand's significand has at least
//     32 trailing zeros (see make_lean), so the sticky bits are not needed;
//   - the shift moves before the product: whether ma * mc reaches 2^105 is
//     one compare of ma with a constant (ceil(2^105 / mc)), and it selects
//     the constant's significand shifted by 9 or by 10.  The product of that
//     with ma << 2 always has its leading bit at bit 116, so its 53 bits
//     are whole words from bit 64 up and the rounding is a carry out of the
//     word below;
//   - that carry, the significand and the sign/exponent word then go
//     together in one three-word add.
#pragma once

#include <cmath>

#include "dpemu.cuh"

namespace qslc {
namespace emu {

// A multiplier fixed for a whole kernel: two 16-byte words.
struct alignas(16) LeanK {
    uint32_t h0, h1;      // mc << 9, when ma * mc >= 2^105
    uint32_t l0, l1;      // mc << 10, when it is below
    uint32_t t0, t1;      // the least ma << 2 with ma * mc >= 2^105
    uint32_t k;           // sign of c and (e(c) - 1) << 20, to be added to the operand's sign/exponent word
    int usable;
};

// ceil(2^105 / m) for a significand m: the IEEE quotient is the nearest
// integer to it, low by at most one.
QSLC_HD uint64_t ceil_2_105(uint64_t m)
{
#ifdef __CUDA_ARCH__
    uint64_t q = uint64_t(__ddiv_rn(0x1p105, double((long long)m)));
#else
    uint64_t q = uint64_t(0x1p105 / double(m));
#endif
    return umulhi(q, m) >= (uint64_t(1) << 41) ? q : q + 1;
}

QSLC_HD LeanK make_lean(double c)
{
    LeanK r{};
    const MulK m = make_mulk(c);
    const uint64_t mc = (dbits(c) & MANT) | HIDDEN;
    // ma * mc is a tie only when its trailing zeros number 51 or 52: with
    // fewer than 20 of them in mc, only for an ma with 32 or more
    r.usable = m.usable && (mc & ((uint64_t(1) << 20) - 1)) != 0;
    r.h0 = uint32_t(mc << 9);
    r.h1 = uint32_t((mc << 9) >> 32);
    r.l0 = uint32_t(mc << 10);
    r.l1 = uint32_t((mc << 10) >> 32);
    const uint64_t t = ceil_2_105(mc) << 2;
    r.t0 = uint32_t(t);
    r.t1 = uint32_t(t >> 32);
    r.k = m.ehi + m.sign;
    return r;
}

// The same for a gate's constants, powers of two included (the sines and cosines
// of quarter turns): a product by a power of two keeps the operand's significand,
// so it is never a tie.
QSLC_HD LeanK make_lean_gate(double c)
{
    LeanK r = make_lean(c);
    r.usable |= make_mulk(c).usable && (dbits(c) & MANT) == 0;
    return r;
}

// The parts of an easy operand that its products share.
struct LeanOp {
    uint32_t lo, hi;      // ma << 2
    uint32_t se;          // sign and exponent field, in place
};

QSLC_HD uint32_t shl2_hi(uint32_t lo, uint32_t hi)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, 2);
#else
    return (hi << 2) | (lo >> 30);
#endif
}

QSLC_HD uint32_t mulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return uint32_t((uint64_t(a) * b) >> 32);
#endif
}

QSLC_HD LeanOp lean_operand(uint64_t a)
{
    const uint32_t ahi = uint32_t(a >> 32), alo = uint32_t(a);
    LeanOp o;
    o.lo = alo << 2;
    o.hi = (shl2_hi(alo, ahi) & 0x003FFFFFu) | 0x00400000u;
    o.se = ahi & 0xFFF00000u;
    return o;
}

// Whether an operand is in the exponent range (the low significand word is
// tested on its own, where it matters).
QSLC_HD bool easy_range(uint64_t a)
{
    const uint32_t ahi = uint32_t(a >> 32);
    return (ahi + ahi) - 2 * PACK_EF_LO20 <= 2 * PACK_EF_SPAN20 + 0x001FFFFFu;
}
QSLC_HD bool easy_product(uint64_t a) { return easy_range(a) & (uint32_t(a) != 0); }

// ---- zeros --------------------------------------------------------------------
// An operand that is easy or a zero of either sign.  A zero has a significand
// of 0 and an exponent of 0: its product has no significand either, and the sign
// alone where the constant's exponent is left out.
struct LeanOpZ {
    LeanOp op;
    bool zero;
};

// By words: the compiler turns a test of the whole into a comparison on the FP64
// pipe, which the sums need (8 comparisons beside the 4 sums of a pair).
QSLC_HD bool is_zero(uint64_t a)
{
    const uint32_t ahi = uint32_t(a >> 32);
    return ((ahi + ahi) | uint32_t(a)) == 0;
}

QSLC_HD LeanOpZ lean_operand_z(uint64_t a)
{
    LeanOpZ o;
    o.op = lean_operand(a);
    o.zero = is_zero(a);
    if (o.zero) o.op.hi = 0;
    return o;
}

// The sign of a constant, in place: its exponent's part of k is negative.
QSLC_HD uint32_t lean_sign(const LeanK &c) { return ~c.k & 0x80000000u; }

// ---- squares ------------------------------------------------------------------
// m * m of a significand m lies in [2^104, 2^106).  It is half-way between two
// doubles only when it has 51 or 52 trailing zeros, m then 26: an operand with
// one of its low 25 bits set rounds on the next bit alone.  The exponent field
// is 512 to 1533, so that the square is normal.
QSLC_HD bool easy_square(uint64_t a)
{
    const uint32_t h = uint32_t(a >> 32) & 0x7FFFFFFFu;
    return ((h - (512u << 20)) < (1022u << 20)) & ((uint32_t(a) & 0x1FFFFFFu) != 0);
}

// The bits of RN(a * a).
QSLC_HD uint64_t lean_square(uint64_t a)
{
    const uint32_t h = uint32_t(a >> 32) & 0x7FFFFFFFu;
    const uint32_t ml = uint32_t(a), mh = (h & 0xFFFFFu) | 0x100000u;
    const uint64_t t0 = uint64_t(ml) * ml;
    const uint64_t t1 = uint64_t(ml) * (2 * mh) + (t0 >> 32);
    const uint64_t t2 = uint64_t(mh) * mh + (t1 >> 32);          // t2 : low word of t1 : low word of t0
    const uint32_t top = uint32_t(t2 >> 41);                     // 1: from 2^105 up
    const uint32_t left = 12 - top, w1 = uint32_t(t1), w0 = uint32_t(t0);
    const uint64_t sig = (t2 << left) | (w1 >> (32 - left));
    const uint32_t half = ((w1 << left) | (w0 >> (32 - left))) >> 31;
    // exponent field 2 E - 1023 + top, less one for the hidden bit
    const uint32_t ex = ((h & 0x7FF00000u) << 1) - (1024u << 20) + (top << 20);
    return sig + (uint64_t(ex) << 32) + half;
}

// (r2:r1:r0) + (k:s1:s0), the top two words: one carry chain.
QSLC_HD uint64_t round96(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t s0, uint32_t s1, uint32_t k, uint32_t &rest)
{
#ifdef __CUDA_ARCH__
    uint32_t lo, hi;
    asm("add.cc.u32 %0, %3, %4;\n\t"
        "addc.cc.u32 %1, %5, %6;\n\t"
        "addc.u32 %2, %7, %8;"
        : "=&r"(rest), "=&r"(lo), "=r"(hi)
        : "r"(r0), "r"(s0), "r"(r1), "r"(s1), "r"(r2), "r"(k));
    return (uint64_t(hi) << 32) | lo;
#else
    const uint64_t t0 = uint64_t(r0) + s0;
    rest = uint32_t(t0);
    const uint64_t t1 = uint64_t(r1) + s1 + (t0 >> 32);
    return (uint64_t(uint32_t(r2 + k + uint32_t(t1 >> 32))) << 32) | uint32_t(t1);
#endif
}

// RN(a * c), packed; k0: the constant's sign and exponent.
QSLC_HD uint64_t lean_mul(const LeanOp &a, const LeanK &c, uint32_t k0)
{
    const bool top = ((uint64_t(a.hi) << 32) | a.lo) >= ((uint64_t(c.t1) << 32) | c.t0);
    const uint32_t c0 = top ? c.h0 : c.l0, c1 = top ? c.h1 : c.l1;
    const uint32_t k = k0 + a.se + (top ? 0x00100000u : 0u);
    // partial sums stay below 2^64: c1 < 2^31, a.hi < 2^23
    const uint64_t mid = mulwide(a.hi, c0) + (mulwide(a.lo, c1) + 0x80000000u);
    const uint64_t high = mulwide(a.hi, c1);
    uint32_t rest;
    return round96(uint32_t(mid), uint32_t(high), uint32_t(high >> 32), mulhi32(a.lo, c0), uint32_t(mid >> 32), k,
                   rest);
}
QSLC_HD uint64_t lean_mul(const LeanOp &a, const LeanK &c) { return lean_mul(a, c, c.k); }
QSLC_HD uint64_t lean_mul(const LeanOpZ &a, const LeanK &c) { return lean_mul(a.op, c, a.zero ? lean_sign(c) : c.k); }

// A divisor fixed for a whole kernel: the reciprocals 2^146 / my (for
// mx >= my) and 2^147 / my (for mx < my), rounded down, as three words.
struct LeanDiv {
    uint32_t h0, h1, h2, l0, l1, l2;
    uint32_t t0, t1;      // my << 2
    uint32_t kh, kl;      // sign of y, and (-e(y) + 1022 + top) << 20 less the operand's bias
    int usable;
};

inline LeanDiv make_lean_div(double y)
{
    LeanDiv r{};
    const DivConst d = make_div(y);
    const uint64_t my = d.m;
    auto recip = [my](int bits, uint32_t *w) {      // floor(2^bits / my), 145 <= bits <= 159
        unsigned __int128 rem = 0;
        uint32_t q[5];
        for (int i = 0; i < 5; i++) {
            const uint32_t digit = (bits / 32 == 4 - i) ? uint32_t(1) << (bits % 32) : 0u;
            const unsigned __int128 cur = (rem << 32) | digit;
            q[i] = uint32_t(cur / my);
            rem = cur % my;
        }
        w[0] = q[4];
        w[1] = q[3];
        w[2] = q[2];
        return (q[0] | q[1]) == 0 && q[2] < 0x80000000u && q[3] < 0xFF000000u;   // see lean_div's bounds
    };
    uint32_t h[3], l[3];
    const bool fits = recip(146, h) & recip(147, l);
    r.h0 = h[0], r.h1 = h[1], r.h2 = h[2];
    r.l0 = l[0], r.l1 = l[1], r.l2 = l[2];
    r.t0 = uint32_t(my << 2);
    r.t1 = uint32_t((my << 2) >> 32);
    // quotient exponent field ef - e(y) - (mx < my), less one for the hidden bit
    r.kh = (uint32_t(-d.e - 1) << 20) + uint32_t(d.sign >> 32);
    r.kl = r.kh - 0x00100000u;
    // exponent fields 65 to 2044 divide to normal quotients for |e(y)| <= 1
    r.usable = d.usable && fits && d.e >= -1 && d.e <= 1;
    return r;
}

// RN(x / y), packed, for an operand in the exponent range; `sure` is
// cleared when the quotient's fraction is too close to one half to decide.
// With R the reciprocal, A = mx << 2, the quotient significand is the part
// of A * R from bit 96 up and the word below it decides the rounding.  The
// sum leaves out A.lo * r0 and the low words of A.lo * r1 and A.hi * r0, so
// the word is low by less than four units, and R's own rounding adds less
// than one.
QSLC_HD uint64_t lean_div(const LeanOp &a, const LeanDiv &y, bool &sure)
{
    const bool top = ((uint64_t(a.hi) << 32) | a.lo) >= ((uint64_t(y.t1) << 32) | y.t0);
    const uint32_t r0 = top ? y.h0 : y.l0, r1 = top ? y.h1 : y.l1, r2 = top ? y.h2 : y.l2;
    const uint32_t k = (top ? y.kh : y.kl) + a.se;
    // r1 < 2^32 - 2^24 and a.hi < 2^23: the sum of the two high words fits
    const uint32_t low = mulhi32(a.lo, r1) + mulhi32(a.hi, r0);
    const uint64_t mid = mulwide(a.hi, r1) + (mulwide(a.lo, r2) + 0x80000000u);
    const uint64_t high = mulwide(a.hi, r2);
    uint32_t rest;
    const uint64_t q =
        round96(uint32_t(mid), uint32_t(high), uint32_t(high >> 32), low, uint32_t(mid >> 32), k, rest);
    sure = sure & (rest + 8u > 8u);
    return q;
}

// RN(x / d) in binary32 for a constant d, r = RN(1 / d), by Markstein's final
// step (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): q within an ulp of the quotient, its exact
// remainder, and one fused correction.  Zeros keep their sign in this
// arrangement of the signs.  Takes zeros and magnitudes from 2^-100 up
// (div_step_takes); the others go to the divide instruction sequence.
QSLC_HD float div_step(float x, float d, float r)
{
#ifdef __CUDA_ARCH__
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(q, d, -x), -r, q);
#else
    volatile float q = x * r;
    return std::fma(std::fma(float(q), d, -x), -r, float(q));
#endif
}
QSLC_HD bool div_step_takes(float x)
{
    const float m = x < 0.f ? -x : x;
    return m == 0.f || (m >= 0x1p-100f && m <= 0x1.fffffep127f);
}

}  // namespace emu
}  // namespace qslc
