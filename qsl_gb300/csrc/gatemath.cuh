// gatemath.cuh -- the arithmetic of one gate output, shared by the plain
// sweeps (gates.cu) and the number-preserving sweeps (np.cu).
//
// Every output is computed as the reference computes it, operation for
// operation, with each product and sum rounded on its own (no FMA).  For
// complex128 an output can instead run on the integer pipes through the
// exact binary64 emulation of dpemu.cuh; the bits are the same either way,
// and the split between the FP64 pipe and the integer pipes is chosen per
// sweep item by a pattern of masks.
#pragma once

#include "qslc_internal.cuh"
#include "dpemu.cuh"
#include "lean.cuh"

#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <type_traits>

namespace qslc {

template <class T>
struct Coef {
    T c, s;  // cos/sin of angle/2 (rotations) or of angle (phase); sqrt2 for H
    emu::MulK mc, ms;       // c and s decoded for the integer products of the mixed path (double only)
    emu::MulConst kc, ks;   // c and s decoded for the full integer path
    emu::DivConst kd;       // c as a divisor (Hadamard)
    emu::LeanK lc, ls;      // c and s for easy operands (lean.cuh)
    emu::LeanDiv ld;        // c as a divisor of easy operands
};

// How one gate output RN(RN(a*k1) +- RN(b*k2)) is computed (complex128):
//   MD_F  both products and the sum on the FP64 pipe (3 FP64 operations);
//   MD_P  both products on the integer pipes (prod_pack), the sum on the
//        FP64 pipe (1 FP64 operation);
//   MD_Q  the first product on the integer pipes, the second product and the
//        sum on the FP64 pipe (2 FP64 operations);
//   MD_E  all of it on the integer pipes (dot2_rn, no FP64 operation).
// Every mode gives the reference's bits; they differ only in which pipes
// they load.  A mode mask holds 2 bits per output.
enum OutMode : unsigned { MD_F = 0, MD_P = 1, MD_Q = 2, MD_E = 3 };

// The FP64 fallbacks of the emulated outputs, out of line.  They run only
// for the operands the integer path declines (subnormals, infinities, NaNs,
// results outside the normal range).  Inline, a fallback of a few FP64
// instructions is cheap enough that the compiler predicates it instead of
// branching around it; predicated FP64 instructions still take their turn
// on the FP64 pipe, so every thread would pay for them and the emulation
// would save nothing.  A call is not turned into predicated arithmetic:
// measured on GB300, the inline forms ran the emulated patterns at the
// all-FP64 speed, the out-of-line form at the speed the pattern predicts.
template <bool NEG>
__device__ __noinline__ double dot2_fallback(double a, double k1, double b, double k2)
{
    return NEG ? __dsub_rn(__dmul_rn(a, k1), __dmul_rn(b, k2)) : __dadd_rn(__dmul_rn(a, k1), __dmul_rn(b, k2));
}
template <bool NEG>
__device__ __noinline__ double hdiv_fallback(double a, double b, double d)
{
    return __ddiv_rn(NEG ? __dsub_rn(a, b) : __dadd_rn(a, b), d);
}

// One Hadamard output, RN(RN(a +- b) / sqrt2) (gates.cpp:95-98).  The
// division always runs on the integer pipes (an FP64 divide is a long
// iteration on the FP64 pipe); with `em` set the sum does too.
template <class T, bool NEG>
__device__ __forceinline__ T hdiv(bool em, T a, T b, const Coef<T> &k)
{
    using R = rn<T>;
    if constexpr (sizeof(T) == 8) {
        bool ok = k.kd.usable != 0;
        if (ok) {
            uint64_t q;
            if (em) {
                const emu::Unp x = emu::unpack(emu::dbits(a), ok);
                emu::Unp y = emu::unpack(emu::dbits(b), ok);
                if (NEG) y.sign ^= emu::SIGN;
                q = emu::div_unp(emu::add_core(x, y, ok), k.kd, ok);
            } else {
                q = emu::div_fast(emu::dbits(NEG ? R::sub(a, b) : R::add(a, b)), k.kd, ok);
            }
            if (ok) return emu::dfrom(q);
        }
        return hdiv_fallback<NEG>(a, b, k.c);
    } else {
        return R::div(NEG ? R::sub(a, b) : R::add(a, b), k.c);
    }
}

// One output of a rotation or phase update: RN(RN(a*k1) + RN(b*k2)), or
// RN(RN(a*k1) - RN(b*k2)) when NEG.  With `em` set the integer pipes compute it
// (dpemu.cuh), falling back to the FP64 pipe for operands the integer path
// declines; either way the bits are the reference's.
template <class T, bool NEG>
__device__ __forceinline__ T dot2(bool em, T a, T k1, const emu::MulConst &e1, T b, T k2,
                                  const emu::MulConst &e2)
{
    if constexpr (sizeof(T) == 8) {
        if (em) {
            bool ok = (e1.usable & e2.usable) != 0;
            const uint64_t r = emu::dot2_rn(emu::dbits(a), e1, emu::dbits(b), e2, NEG, ok);
            if (ok) return emu::dfrom(r);
            return dot2_fallback<NEG>(a, k1, b, k2);
        }
    }
    using R = rn<T>;
    return NEG ? R::sub(R::mul(a, k1), R::mul(b, k2)) : R::add(R::mul(a, k1), R::mul(b, k2));
}

// One output in the given mode (see OutMode); `mode` must be the same
// across a warp.  Operands the integer products decline go to the FP64
// pipe out of line, as in dot2.
template <class T, bool NEG>
__device__ __forceinline__ T dot2m(unsigned mode, T a, T k1, const emu::MulConst &e1, const emu::MulK &m1,
                                   T b, T k2, const emu::MulConst &e2, const emu::MulK &m2)
{
    if constexpr (sizeof(T) == 8) {
        if (mode == MD_E) return dot2<T, NEG>(true, a, k1, e1, b, k2, e2);
        if (mode == MD_P) {
            bool ok = (m1.usable & m2.usable) != 0;
            const double p = emu::dfrom(emu::prod_pack(emu::dbits(a), m1, ok));
            const double q = emu::dfrom(emu::prod_pack(emu::dbits(b), m2, ok));
            if (ok) return NEG ? __dsub_rn(p, q) : __dadd_rn(p, q);
            return dot2_fallback<NEG>(a, k1, b, k2);
        }
        if (mode == MD_Q) {
            bool ok = m1.usable != 0;
            const double p = emu::dfrom(emu::prod_pack(emu::dbits(a), m1, ok));
            if (ok) {
                const double q = __dmul_rn(b, k2);
                return NEG ? __dsub_rn(p, q) : __dadd_rn(p, q);
            }
            return dot2_fallback<NEG>(a, k1, b, k2);
        }
    }
    using R = rn<T>;
    return NEG ? R::sub(R::mul(a, k1), R::mul(b, k2)) : R::add(R::mul(a, k1), R::mul(b, k2));
}

enum PairOp { P_SWAP, P_Y, P_H, P_RX, P_RY, P_RZ };
enum DiagOp { D_NEG, D_PHASE, D_PHASE_INV };   // D_PHASE_INV: s with its sign flipped (the NP rotateZ)

// Output i of a pair (r0.x, r0.y, r1.x, r1.y) takes mode (md >> 2i) & 3;
// Hadamard's sums run on the integer pipes for any mode but MD_F.  `md`
// must be the same across a warp.
__host__ __device__ constexpr unsigned mode_of(unsigned md, int i) { return (md >> (2 * i)) & 3u; }

template <class T, int OP>
__device__ __forceinline__ void pair_update(cplx<T> &a0, cplx<T> &a1, const Coef<T> &k, unsigned md = 0)
{
    using R = rn<T>;
    cplx<T> r0, r1;
    const unsigned E0 = mode_of(md, 0), E1 = mode_of(md, 1), E2 = mode_of(md, 2), E3 = mode_of(md, 3);
    if constexpr (OP == P_SWAP) {            // gates.cpp:41, :236, :524
        r0 = a1;
        r1 = a0;
    } else if constexpr (OP == P_Y) {        // gates.cpp:59-62, :267-270
        r0.x = a1.y; r0.y = -a1.x;
        r1.x = -a0.y; r1.y = a0.x;
    } else if constexpr (OP == P_H) {        // gates.cpp:95-98, :493-496, :675-678
        r0.x = hdiv<T, false>(E0 != MD_F, a0.x, a1.x, k);
        r0.y = hdiv<T, false>(E1 != MD_F, a0.y, a1.y, k);
        r1.x = hdiv<T, true>(E2 != MD_F, a0.x, a1.x, k);
        r1.y = hdiv<T, true>(E3 != MD_F, a0.y, a1.y, k);
    } else if constexpr (OP == P_RX) {       // gates.cpp:139-144, :336-341, :595-600
        r0.x = dot2m<T, false>(E0, a0.x, k.c, k.kc, k.mc, a1.y, k.s, k.ks, k.ms);
        r0.y = dot2m<T, true>(E1, a0.y, k.c, k.kc, k.mc, a1.x, k.s, k.ks, k.ms);
        r1.x = dot2m<T, false>(E2, a1.x, k.c, k.kc, k.mc, a0.y, k.s, k.ks, k.ms);
        r1.y = dot2m<T, true>(E3, a1.y, k.c, k.kc, k.mc, a0.x, k.s, k.ks, k.ms);
    } else if constexpr (OP == P_RY) {       // gates.cpp:169-174, :380-385, :638-643
        r0.x = dot2m<T, true>(E0, a0.x, k.c, k.kc, k.mc, a1.x, k.s, k.ks, k.ms);
        r0.y = dot2m<T, true>(E1, a0.y, k.c, k.kc, k.mc, a1.y, k.s, k.ks, k.ms);
        r1.x = dot2m<T, false>(E2, a0.x, k.s, k.ks, k.ms, a1.x, k.c, k.kc, k.mc);
        r1.y = dot2m<T, false>(E3, a0.y, k.s, k.ks, k.ms, a1.y, k.c, k.kc, k.mc);
    } else {                                 // P_RZ: gates.cpp:200-205, :424-429
        r0.x = dot2m<T, false>(E0, a0.x, k.c, k.kc, k.mc, a0.y, k.s, k.ks, k.ms);
        r0.y = dot2m<T, true>(E1, a0.y, k.c, k.kc, k.mc, a0.x, k.s, k.ks, k.ms);
        r1.x = dot2m<T, true>(E2, a1.x, k.c, k.kc, k.mc, a1.y, k.s, k.ks, k.ms);
        r1.y = dot2m<T, false>(E3, a1.y, k.c, k.kc, k.mc, a1.x, k.s, k.ks, k.ms);
    }
    a0 = r0;
    a1 = r1;
}

// Output i of a diagonal update (x, y) takes mode (md >> 2i) & 3.
template <class T, int OP>
__device__ __forceinline__ void diag_update(cplx<T> &a, const Coef<T> &k, unsigned md = 0)
{
    using R = rn<T>;
    if constexpr (OP == D_NEG) {             // gates.cpp:76-77, :296-297 (x *= -1)
        a.x = R::mul(a.x, T(-1));
        a.y = R::mul(a.y, T(-1));
    } else {                                 // gates.cpp:114-115, :460-461
        T x = a.x, y = a.y;
        a.x = dot2m<T, true>(mode_of(md, 0), x, k.c, k.kc, k.mc, y, k.s, k.ks, k.ms);
        a.y = dot2m<T, false>(mode_of(md, 1), y, k.c, k.kc, k.mc, x, k.s, k.ks, k.ms);
    }
}

// ---------------------------------------------------------------------------
// Updates of easy operands (lean.cuh): products and divisions on the integer
// pipes, one FP64 add per output.  Each returns whether it ran; when it did
// not, the amplitudes are unchanged and the caller takes the general update.
// Each thread decides for itself, with no vote: the updates are called from
// divergent code (items past a sweep's end, controls tested per thread), where
// no mask is known that names exactly the lanes of a vote.
//
// Bound by the FP64 pipe (two operations per SM and clock) and the ALU pipe
// together: 100 instructions per amplitude and gate against 150 with the
// general split "PPPQ", 2 of them FP64 instead of 2.7.  Two rotateX gates of a
// 26-qubit dense state in one sweep: 761 us with the general split, 550 us
// with this; FP64 pipe 79% busy.
//
// Three forms, from the cheapest: easy operands; operands that are easy or
// zero; any.  Constants may be powers of two (make_lean_gate), so quarter turns
// are easy too: two rotateX(pi) 885 us without, 550 with.
// ---------------------------------------------------------------------------
// Every rotation and phase is made of turns of two parts (u, v) to
// (u c - v s, v c + u s), with s negated for INV: rotateX turns (a0.x, a1.y) and
// (a1.x, a0.y), rotateY (a0.x, a1.x) and (a0.y, a1.y), rotateZ and phase the
// parts of one amplitude.  `flip` (0x80000000 or 0) negates s at run time.
template <class Op>
__device__ __forceinline__ double lean_prod(const Op &a, const emu::LeanK &k, uint32_t flip = 0)
{
    return emu::dfrom(emu::lean_mul(a, k) ^ (uint64_t(flip) << 32));
}
template <bool INV, class Op>
__device__ __forceinline__ void turn(double &u, double &v, const Op &a, const Op &b, const emu::LeanK &lc,
                                     const emu::LeanK &ls, uint32_t flip)
{
    const double uc = lean_prod(a, lc), vs = lean_prod(b, ls, flip), vc = lean_prod(b, lc), us = lean_prod(a, ls, flip);
    u = INV ? __dadd_rn(uc, vs) : __dsub_rn(uc, vs);
    v = INV ? __dsub_rn(vc, us) : __dadd_rn(vc, us);
}
template <bool INV>
__device__ __forceinline__ void turn_easy(double &u, double &v, const emu::LeanK &lc, const emu::LeanK &ls,
                                          uint32_t flip = 0)
{
    turn<INV>(u, v, emu::lean_operand(emu::dbits(u)), emu::lean_operand(emu::dbits(v)), lc, ls, flip);
}
__device__ __forceinline__ double zero_of(uint32_t sign)
{
    return __hiloint2double(int(sign & 0x80000000u), 0);
}
// The turn of two zeros: a sum of two zeros is -0 when both are, a difference
// p - q when p is -0 and q is +0.  csign, ssign: the signs of c and s.
template <bool INV>
__device__ __forceinline__ void turn_signs(double &u, double &v, uint32_t csign, uint32_t ssign)
{
    const uint32_t a = uint32_t(__double2hiint(u)), b = uint32_t(__double2hiint(v)), t = INV ? ssign : ~ssign;
    u = zero_of((a ^ csign) & (b ^ t));
    v = zero_of((b ^ csign) & (a ^ ~t));
}
// The turn of parts that are easy or zeros: the zeros of a real state's imaginary
// parts, say, only take signs.
template <bool INV>
__device__ __forceinline__ void turn_zeros(double &u, double &v, const emu::LeanK &lc, const emu::LeanK &ls,
                                           uint32_t flip = 0)
{
    const uint64_t a = emu::dbits(u), b = emu::dbits(v);
    if (emu::is_zero(a) & emu::is_zero(b)) turn_signs<INV>(u, v, emu::lean_sign(lc), emu::lean_sign(ls) ^ flip);
    else turn<INV>(u, v, emu::lean_operand_z(a), emu::lean_operand_z(b), lc, ls, flip);
}

template <int OP, class F, class G>
__device__ __forceinline__ void pair_turns(double2 &a0, double2 &a1, F &&turn_inv, G &&turn_fwd)
{
    if constexpr (OP == P_RX) {
        turn_inv(a0.x, a1.y);
        turn_inv(a1.x, a0.y);
    } else if constexpr (OP == P_RY) {
        turn_fwd(a0.x, a1.x);
        turn_fwd(a0.y, a1.y);
    } else {
        turn_inv(a0.x, a0.y);
        turn_fwd(a1.x, a1.y);
    }
}

__device__ __forceinline__ bool takes(double v) { return emu::easy_product(emu::dbits(v)); }
__device__ __forceinline__ bool takes_zero(double v) { return takes(v) | emu::is_zero(emu::dbits(v)); }
__device__ __forceinline__ bool zeros(const double2 &a)
{
    return emu::is_zero(emu::dbits(a.x)) & emu::is_zero(emu::dbits(a.y));
}
__device__ __forceinline__ bool takes(const double2 &a) { return takes(a.x) & takes(a.y); }
__device__ __forceinline__ bool takes_zero(const double2 &a) { return takes_zero(a.x) & takes_zero(a.y); }

template <int OP>
__device__ __forceinline__ bool pair_lean(double2 &a0, double2 &a1, const emu::LeanK &lc, const emu::LeanK &ls)
{
    if (!((lc.usable & ls.usable) != 0 && takes(a0) & takes(a1))) return false;
    pair_turns<OP>(a0, a1, [&](double &u, double &v) { turn_easy<true>(u, v, lc, ls); },
                   [&](double &u, double &v) { turn_easy<false>(u, v, lc, ls); });
    return true;
}
template <int OP>
__device__ __forceinline__ bool pair_zeros(double2 &a0, double2 &a1, const emu::LeanK &lc, const emu::LeanK &ls)
{
    if (!((lc.usable & ls.usable) != 0 && takes_zero(a0) & takes_zero(a1))) return false;
    pair_turns<OP>(a0, a1, [&](double &u, double &v) { turn_zeros<true>(u, v, lc, ls); },
                   [&](double &u, double &v) { turn_zeros<false>(u, v, lc, ls); });
    return true;
}
template <bool INV>
__device__ __forceinline__ bool phase_lean(double2 &a, const emu::LeanK &lc, const emu::LeanK &ls, uint32_t flip = 0)
{
    if (!((lc.usable & ls.usable) != 0 && takes(a))) return false;
    turn_easy<INV>(a.x, a.y, lc, ls, flip);
    return true;
}
template <bool INV>
__device__ __forceinline__ bool phase_zeros(double2 &a, const emu::LeanK &lc, const emu::LeanK &ls, uint32_t flip = 0)
{
    if (!((lc.usable & ls.usable) != 0 && takes_zero(a))) return false;
    turn_zeros<INV>(a.x, a.y, lc, ls, flip);
    return true;
}

// Hadamard's quotients of the sums s and differences d by sqrt(2).
__device__ __forceinline__ bool quotients_lean(double2 &s, double2 &d, const emu::LeanDiv &ld)
{
    const uint64_t b0 = emu::dbits(s.x), b1 = emu::dbits(s.y), b2 = emu::dbits(d.x), b3 = emu::dbits(d.y);
    if (!(ld.usable && emu::easy_range(b0) & emu::easy_range(b1) & emu::easy_range(b2) & emu::easy_range(b3)))
        return false;
    bool sure = true;
    const uint64_t q0 = emu::lean_div(emu::lean_operand(b0), ld, sure);
    const uint64_t q1 = emu::lean_div(emu::lean_operand(b1), ld, sure);
    const uint64_t q2 = emu::lean_div(emu::lean_operand(b2), ld, sure);
    const uint64_t q3 = emu::lean_div(emu::lean_operand(b3), ld, sure);
    if (!sure) return false;
    s = make_double2(emu::dfrom(q0), emu::dfrom(q1));
    d = make_double2(emu::dfrom(q2), emu::dfrom(q3));
    return true;
}
// The same with zeros, their own quotients: a part whose sum and difference are zeros
// (a real state's imaginary one) is left as it is.  False, with the values
// unchanged, when one needs the general division.
__device__ __forceinline__ bool quotients_zeros(double2 &s, double2 &d, const emu::LeanDiv &ld)
{
    bool sure = ld.usable != 0;
    double2 qs = s, qd = d;
    auto part = [&](double &x, double &y) {
        const uint64_t a = emu::dbits(x), b = emu::dbits(y);
        const bool za = emu::is_zero(a), zb = emu::is_zero(b);
        if (za & zb) return;
        sure = sure & (za | emu::easy_range(a)) & (zb | emu::easy_range(b));
        bool sa = true, sb = true;
        const double u = emu::dfrom(emu::lean_div(emu::lean_operand(a), ld, sa));
        const double v = emu::dfrom(emu::lean_div(emu::lean_operand(b), ld, sb));
        sure = sure & (za | sa) & (zb | sb);
        x = za ? x : u;
        y = zb ? y : v;
    };
    part(qs.x, qd.x);
    part(qs.y, qd.y);
    if (!sure) return false;
    s = qs;
    d = qd;
    return true;
}

// The old single-bit masks (bit i set: output i fully on the integer pipes)
// as a mode mask.
__host__ __device__ constexpr unsigned modes_from_bits(unsigned em)
{
    return ((em & 1u) ? 3u : 0u) | ((em & 2u) ? 12u : 0u) | ((em & 4u) ? 48u : 0u) | ((em & 8u) ? 192u : 0u);
}

// Bit insertion in the index type of a sweep: 32-bit arithmetic for states
// of up to 31 qubits (every index and shift then fits), 64-bit above.
template <class IX>
__host__ __device__ __forceinline__ IX ins0(IX j, unsigned t)
{
    const IX low = j & ((IX(1) << t) - 1);
    return ((j >> t) << (t + 1)) | low;
}
template <class IX>
__host__ __device__ __forceinline__ IX ins00(IX j, unsigned lo, unsigned hi)
{
    return ins0<IX>(ins0<IX>(j, lo), hi);
}

// The sweeps below take ITEMS work items per grid-stride iteration (at j,
// j + stride, j + 2 stride), all loads first.  `pat` holds one emulation
// mask per item, 4 bits each: item r uses (pat >> 4r) & 15, so the share of
// outputs computed on the integer pipes can be set in steps of one output
// in twelve (pair gates) or one in six (diagonal gates).  Masks differ only
// between items, never between threads of a warp.
#ifndef QSLC_ITEMS
#define QSLC_ITEMS 3
#endif
constexpr int ITEMS = QSLC_ITEMS;
// The easy form (PAT_LEAN) has its own shape: items per iteration for pair
// gates and diagonal gates, and CTAs of 256 threads per SM.
// Measured on a dense 28-qubit state, TB/s of algorithmic bytes, rotateX /
// phase: 1 item 6.12 / 5.23, 2 items 6.62 / 5.56, 3 items 6.53 / 5.79, 4
// items - / 6.11 (four CTAs); rotateX with 2 items 6.25 on three CTAs and
// 6.43 on five.  Hadamard of a 26-qubit state takes 332 us with two items, 370
// with one.
#ifndef QSLC_LEAN_ITEMS
#define QSLC_LEAN_ITEMS 2
#endif
#ifndef QSLC_LEAN_ITEMS_D
#define QSLC_LEAN_ITEMS_D 4
#endif
#ifndef QSLC_LEAN_CTAS
#define QSLC_LEAN_CTAS 4
#endif

// Launch bounds of the sweep kernels: 256 threads, and with QSLC_MINB set,
// at least that many resident CTAs per SM (which caps the registers).
#if defined(QSLC_MINB) && QSLC_MINB > 0
#define QSLC_SWEEP_BOUNDS __launch_bounds__(256, QSLC_MINB)
#else
#define QSLC_SWEEP_BOUNDS __launch_bounds__(256)
#endif
#define QSLC_LEAN_BOUNDS(CPAT) __launch_bounds__(256, (CPAT) == PAT_LEAN ? QSLC_LEAN_CTAS : 1)

// A kernel's pattern is a template argument where it is compiled in (the
// mask tests then fold away, and so do the unused arithmetic paths and
// their registers): 0, all on the FP64 pipe, and PAT_LEAN.  PAT_RUNTIME
// takes it from the kernel's argument instead, for any other setting.
constexpr unsigned PAT_RUNTIME = 0xFFFFFFFFu;

// PAT_LEAN, the default of the complex128 sweeps: the easy form first
// (pair_gate, diag_gate), with the default pattern for the operands it leaves.
constexpr unsigned PAT_LEAN = 0xFFFFFFFEu;

// The default splits of the general path.  A pattern holds one 8-bit mode
// mask per sweep item (item r at bits 8r..8r+7), 2 bits per output
// (OutMode): 0x95 is P, P, P, Q for r0.x, r0.y, r1.x, r1.y, and 0x9 is P, Q
// for a diagonal update's x, y.
constexpr unsigned PAT_ROT = 0x959595u;
constexpr unsigned PAT_H = 0u;
constexpr unsigned PAT_DIAG = 0x090909u;

// The operands that the easy form leaves: first the form with zeros, then the
// general update.  Operands that are all +0 (most of a sparse state) only
// need the signs of their zeros, which follow from the signs of the
// coefficients, easy or not.  That holds for finite coefficients: those of an
// infinite or NaN angle are NaN, and so is their product with a zero.
//
// The sweeps of several gates call the general update out of line (pair_slow and
// the like): inline, once per gate type and pair, it would double their code.
// There the coefficients go by address (of a kernel parameter): by value they
// would take registers and stack of every thread.  The sweeps of one gate have it
// inline, where it costs them less than the call's registers: measured at 26
// qubits, controlRotateX 201 against 212 us.
struct SlowCoef {          // the first members of a Coef<double>
    double c, s;
    emu::MulK mc, ms;
};
static_assert(offsetof(Coef<double>, ms) == offsetof(SlowCoef, ms), "SlowCoef heads Coef<double>");
__device__ __forceinline__ const SlowCoef *slow_coef(const Coef<double> &k)
{
    return reinterpret_cast<const SlowCoef *>(&k);
}
__device__ __forceinline__ Coef<double> general_coef(const SlowCoef *q)
{
    Coef<double> k{};
    k.c = q->c;
    k.s = q->s;
    k.mc = q->mc;
    k.ms = q->ms;
    return k;
}
__device__ __forceinline__ bool plus_zero(const double2 &a)
{
    return (emu::dbits(a.x) | emu::dbits(a.y)) == 0;
}
// Whether c and s are finite; the sine and cosine of one angle are finite together.
__device__ __forceinline__ bool finite_coef(const SlowCoef *q)
{
    return (__double2hiint(q->c) & 0x7FF00000) != 0x7FF00000;
}

struct Pair {
    double2 a0, a1;
};
template <int OP>
__device__ __forceinline__ Pair pair_general(double2 a0, double2 a1, const SlowCoef *q)
{
    if (plus_zero(a0) & plus_zero(a1) & finite_coef(q)) {
        const uint32_t c = uint32_t(__double2hiint(q->c)), s = uint32_t(__double2hiint(q->s));
        pair_turns<OP>(a0, a1, [&](double &u, double &v) { turn_signs<true>(u, v, c, s); },
                       [&](double &u, double &v) { turn_signs<false>(u, v, c, s); });
    } else {
        pair_update<double, OP>(a0, a1, general_coef(q), PAT_ROT & 0xFFu);
    }
    return Pair{a0, a1};
}
__device__ __forceinline__ Pair quotients_general(double2 s, double2 d, double r, const emu::DivConst *kd)
{
    auto quotient = [&](double x) {
        bool ok = kd->usable != 0;
        if (ok) {
            const uint64_t q = emu::div_fast(emu::dbits(x), *kd, ok);
            if (ok) return emu::dfrom(q);
        }
        return __ddiv_rn(x, r);
    };
    return Pair{make_double2(quotient(s.x), quotient(s.y)), make_double2(quotient(d.x), quotient(d.y))};
}
// x c - y s, y c + x s (INV: s with its sign flipped)
template <bool INV>
__device__ __forceinline__ double2 phase_general(double2 a, const SlowCoef *q)
{
    const double x = a.x, y = a.y;
    if (plus_zero(a) & finite_coef(q)) {
        turn_signs<INV>(a.x, a.y, uint32_t(__double2hiint(q->c)), uint32_t(__double2hiint(q->s)));
        return a;
    }
    const Coef<double> k = general_coef(q);
    a.x = dot2m<double, !INV>(PAT_DIAG & 3u, x, k.c, k.kc, k.mc, y, k.s, k.ks, k.ms);
    a.y = dot2m<double, INV>((PAT_DIAG >> 2) & 3u, y, k.c, k.kc, k.mc, x, k.s, k.ks, k.ms);
    return a;
}

template <int OP>
__device__ __noinline__ Pair pair_slow(double2 a0, double2 a1, const SlowCoef *q)
{
    return pair_general<OP>(a0, a1, q);
}
static __device__ __noinline__ Pair quotients_slow(double2 s, double2 d, double r, const emu::DivConst *kd)
{
    return quotients_general(s, d, r, kd);
}
template <bool INV>
__device__ __noinline__ double2 phase_slow(double2 a, const SlowCoef *q)
{
    return phase_general<INV>(a, q);
}

// A gate's update of a pair or of one amplitude: the easy form where it runs,
// else the form with zeros, else the general one, out of line for CALL, with the
// coefficients at `q` (`kd` for Hadamard).  Two gates of a 26-qubit state whose
// imaginary parts are zero, us, on the general split without easy operands / with
// the easy form and the general call only / with zeros: rotateY 764, 934, 457;
// Hadamard 539, 1068, 550.  rotateZ leaves out the form with zeros where the
// general one is a call: it meets zeros in single lanes beside easy ones, which
// then run both (1093 us with it, 725 without).
template <int OP, bool CALL = true>
__device__ __forceinline__ void pair_either(double2 &a0, double2 &a1, const Coef<double> &k, const SlowCoef *q,
                                            const emu::DivConst *kd)
{
    if constexpr (OP == P_H) {
        double2 s = make_double2(__dadd_rn(a0.x, a1.x), __dadd_rn(a0.y, a1.y));
        double2 d = make_double2(__dsub_rn(a0.x, a1.x), __dsub_rn(a0.y, a1.y));
        // opaque from here: the compiler would otherwise compute the sums a
        // second time after the test, and the FP64 pipe is what binds
        asm volatile("" : "+d"(s.x), "+d"(s.y), "+d"(d.x), "+d"(d.y));
        if (!quotients_lean(s, d, k.ld) && !quotients_zeros(s, d, k.ld)) {
            const Pair r = CALL ? quotients_slow(s, d, k.c, kd) : quotients_general(s, d, k.c, kd);
            s = r.a0;
            d = r.a1;
        }
        a0 = s;
        a1 = d;
    } else if (!pair_lean<OP>(a0, a1, k.lc, k.ls) && !((!CALL || OP != P_RZ) && pair_zeros<OP>(a0, a1, k.lc, k.ls))) {
        const Pair r = CALL ? pair_slow<OP>(a0, a1, q) : pair_general<OP>(a0, a1, q);
        a0 = r.a0;
        a1 = r.a1;
    }
}
template <bool INV, bool CALL = true>
__device__ __forceinline__ void phase_either(double2 &a, const Coef<double> &k, const SlowCoef *q)
{
    if (!phase_lean<INV>(a, k.lc, k.ls) && !phase_zeros<INV>(a, k.lc, k.ls))
        a = CALL ? phase_slow<INV>(a, q) : phase_general<INV>(a, q);
}
// phase_either with the sign of s chosen at run time.
__device__ __forceinline__ void phase_flip(double2 &a, uint32_t flip, const Coef<double> &k, const SlowCoef *q)
{
    if (!phase_lean<false>(a, k.lc, k.ls, flip) && !phase_zeros<false>(a, k.lc, k.ls, flip))
        a = flip ? phase_slow<true>(a, q) : phase_slow<false>(a, q);
}

// The same for the sweeps of one gate, whose coefficients are a kernel
// parameter; with LEAN false (and for gates without arithmetic) the general
// update alone, in modes `md`.
template <class T, int OP, bool LEAN>
__device__ __forceinline__ void pair_gate(cplx<T> &a0, cplx<T> &a1, const Coef<T> &k, unsigned md)
{
    if constexpr (LEAN && sizeof(T) == 8 && OP != P_SWAP && OP != P_Y)
        pair_either<OP, false>(a0, a1, k, slow_coef(k), &k.kd);
    else
        pair_update<T, OP>(a0, a1, k, md);
}
template <class T, int OP, bool LEAN>
__device__ __forceinline__ void diag_gate(cplx<T> &a, const Coef<T> &k, unsigned md)
{
    if constexpr (LEAN && sizeof(T) == 8 && OP != D_NEG) phase_either<OP == D_PHASE_INV, false>(a, k, slow_coef(k));
    else diag_update<T, OP>(a, k, md);
}

// The mask of item r (the pattern repeats after three) of a sweep compiled
// for CPAT, its general path in pattern DFLT when CPAT is PAT_LEAN.
template <unsigned CPAT, unsigned DFLT>
__device__ __forceinline__ unsigned item_modes(unsigned pat, int r)
{
    const unsigned p = CPAT == PAT_RUNTIME ? pat : CPAT == PAT_LEAN ? DFLT : CPAT;
    return (p >> (8 * (r % 3))) & 0xFFu;
}
template <int OP>
constexpr unsigned pair_pattern() { return OP == P_H ? PAT_H : PAT_ROT; }

template <unsigned CPAT, int LEAN_ITEMS>
constexpr int sweep_items() { return CPAT == PAT_LEAN ? LEAN_ITEMS : ITEMS; }

// Launch `f(std::integral_constant<unsigned, P>{})` with P = PAT_LEAN when
// `lean`, else 0 when pat is 0 (all on the FP64 pipe), else PAT_RUNTIME.
// CHOICE is false where there is no arithmetic to place: P is 0 then.
template <bool CHOICE, class F>
void with_pattern(bool lean, unsigned pat, F &&f)
{
    if constexpr (!CHOICE) f(std::integral_constant<unsigned, 0u>{});
    else if (lean) f(std::integral_constant<unsigned, PAT_LEAN>{});
    else if (pat == 0) f(std::integral_constant<unsigned, 0u>{});
    else f(std::integral_constant<unsigned, PAT_RUNTIME>{});
}

// Host-side coefficients, computed exactly as the reference does: in Fp,
// with std::cos/std::sin of angle/2 (gates.cpp:124-125) or of angle
// (:106), and sqrt2 = Fp(std::sqrt(2)) (:94).
template <class T>
Coef<T> coef(T c, T s)
{
    Coef<T> k{};
    k.c = c;
    k.s = s;
    k.kc = emu::make_const(double(c));
    k.ks = emu::make_const(double(s));
    k.mc = emu::make_mulk(double(c));
    k.ms = emu::make_mulk(double(s));
    k.kd = emu::make_div(double(c));
    k.lc = emu::make_lean_gate(double(c));
    k.ls = emu::make_lean_gate(double(s));
    k.ld = emu::make_lean_div(double(c));
    return k;
}
// The pattern a gate with coefficients k runs: `pat`, unless a coefficient
// is outside the integer products' range (an exact zero, a sine below
// 2^-64), where every output would decline to the FP64 pipe one by one --
// then all outputs run there from the start.
template <class T>
unsigned pattern_for(const Coef<T> &k, unsigned pat)
{
    return (k.mc.usable && k.ms.usable) ? pat : 0u;
}

template <class T>
Coef<T> half_angle(double angle)
{
    T a = T(angle);
    return coef<T>(T(std::cos(a / 2)), T(std::sin(a / 2)));
}
template <class T>
Coef<T> full_angle(double angle)
{
    T a = T(angle);
    return coef<T>(T(std::cos(a)), T(std::sin(a)));
}
template <class T>
Coef<T> sqrt2_coef()
{
    return coef<T>(T(std::sqrt(2)), T(0));
}

// Share of the dense updates' work done on the integer pipes, as a pattern
// of one mode mask per sweep item (see ITEMS and OutMode), where the easy
// form does not run.  The environment variables that override the defaults
// also turn the easy form off: QSLC_EMU_MASK (rotations, one-qubit
// and controlled), QSLC_EMU_MASK_H (Hadamard), QSLC_EMU_MASK_DIAG (phase and
// controlPhase), QSLC_EMU_MASK_NP and QSLC_EMU_MASK_NP_DIAG (the
// number-preserving sweeps).  The value is one item ("PPPQ") or three
// ("PPPP,PPPP,PPPQ"), each a letter per output -- F, P, Q or E, as in
// OutMode -- or a decimal number in the older form (bit i set: output i
// fully on the integer pipes, mode E).  Items left out repeat the last one.
inline unsigned parse_item(const char *c, const char **endp, unsigned outputs, bool &good)
{
    unsigned md = 0;
    if (*c >= '0' && *c <= '9') {
        char *e = nullptr;
        const long v = std::strtol(c, &e, 10);
        *endp = e;
        if (v < 0 || v >= (1L << outputs)) good = false;
        return modes_from_bits(unsigned(v) & ((1u << outputs) - 1));
    }
    unsigned i = 0;
    for (; *c && *c != ','; c++, i++) {
        unsigned m;
        switch (*c) {
        case 'F': case 'f': m = MD_F; break;
        case 'P': case 'p': m = MD_P; break;
        case 'Q': case 'q': m = MD_Q; break;
        case 'E': case 'e': m = MD_E; break;
        default: m = MD_F; good = false; break;
        }
        if (i < outputs) md |= m << (2 * i);
        else good = false;
    }
    if (i == 0) good = false;
    *endp = c;
    return md;
}

inline unsigned parse_pattern(const char *var, const char *dflt, unsigned outputs)
{
    const char *e = std::getenv(var);
    unsigned m[3] = {0, 0, 0};   // three masks whatever ITEMS is; kernels use the first ITEMS
    for (int attempt = 0; attempt < 2; attempt++) {
        const char *src = (attempt == 0 && e && *e) ? e : dflt;
        bool good = true;
        int n = 0;
        for (const char *c = src; *c && n < 3;) {
            const char *endp = c;
            m[n++] = parse_item(c, &endp, outputs, good);
            if (*endp != ',') {
                if (*endp) good = false;
                break;
            }
            c = endp + 1;
        }
        if (n == 0) good = false;
        for (int i = n; i < 3; i++) m[i] = n ? m[n - 1] : 0;
        if (good) break;                 // a malformed override falls back to the default
    }
    return m[0] | (m[1] << 8) | (m[2] << 16);
}
inline unsigned pattern_rot()
{
    static unsigned p = parse_pattern("QSLC_EMU_MASK", "PPPQ", 4);
    return p;
}
// Whether the variable is unset: the sweeps then run PAT_LEAN.
inline bool unset(const char *var)
{
    const char *e = std::getenv(var);
    return !(e && *e);
}
inline bool lean_rot()
{
    static const bool b = unset("QSLC_EMU_MASK");
    return b;
}
inline bool lean_h()
{
    static const bool b = unset("QSLC_EMU_MASK_H");
    return b;
}
inline bool lean_diag()
{
    static const bool b = unset("QSLC_EMU_MASK_DIAG");
    return b;
}
inline bool lean_np_pair()
{
    static const bool b = unset("QSLC_EMU_MASK_NP");
    return b;
}
inline bool lean_np_diag()
{
    static const bool b = unset("QSLC_EMU_MASK_NP_DIAG");
    return b;
}
inline unsigned pattern_h()
{
    static unsigned p = parse_pattern("QSLC_EMU_MASK_H", "FFFF", 4);
    return p;
}
inline unsigned pattern_diag()
{
    static unsigned p = parse_pattern("QSLC_EMU_MASK_DIAG", "PQ", 2);
    return p;
}
// The number-preserving sweeps spend integer work on ranking their indices,
// so their defaults differ: QSLC_EMU_MASK_NP (pair gates) and
// QSLC_EMU_MASK_NP_DIAG (single amplitudes).
inline unsigned pattern_np_pair()
{
    static unsigned p = parse_pattern("QSLC_EMU_MASK_NP", "PPPQ", 4);
    return p;
}
inline unsigned pattern_np_diag()
{
    static unsigned p = parse_pattern("QSLC_EMU_MASK_NP_DIAG", "PQ", 2);
    return p;
}

}  // namespace qslc
