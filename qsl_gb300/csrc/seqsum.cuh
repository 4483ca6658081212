// seqsum.cuh -- bit-exact sequential sums and CDF sampling over a state.
//
// A "producer" describes the sequence the reference sums: element j of
// the sequence is |a|^2 of one stored amplitude, and index(j) is the basis
// index it stands for.  prob(targ, outcome) sums the amplitudes whose bit
// `targ` equals `outcome` in ascending index order (measure.cpp:126-147);
// the sampling CDF sums every amplitude in ascending order
// (measure.cpp:60-78).
//
// The sum is computed on the device, in tiles of SEQ_TILE consecutive
// elements, with one pass over the state and no host step in between:
//   1. k_seq_estimate: an estimate of each tile's sum from a sample of it;
//   2. k_seq_guess: from their prefix sums, a guess of the binade the running
//      sum occupies in each tile;
//   3. k_seq_steps: the effect of each tile on a running sum of that binade,
//      in grid steps (replay.cuh) -- which is also the tile's sum to within
//      rounding;
//   4. k_seq_guess again, on these sums: the tiles whose guess was wrong go on
//      a list, and k_seq_steps does them again;
//   5. k_seq_walk: one CTA walks the tiles in order, a few thousand a round by
//      a scan of their effects, and advances the exact running sum; the few
//      tiles in which it crosses a power of two (or whose guess is still
//      wrong) it walks term by term, in rounds too;
//   6. for sampling, k_seq_shots: one warp per uniform finds the tile, the
//      512-term piece and the term whose partial sum is the first to reach
//      the uniform; the reference's binary search over its Dist vector
//      (measure.cpp:164-188) returns the same element.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "lean.cuh"
#include "qslc_internal.cuh"
#include "replay.cuh"

namespace qslc {

constexpr int SEQ_TILE = 4096;
constexpr int SEQ_TPB = 256;
constexpr int SEQ_PER = SEQ_TILE / SEQ_TPB;
constexpr int SEQ_AHEAD = 4;               // terms a thread of k_seq_steps loads together
constexpr int SEQ_PIECES = SEQ_TPB / 32;   // pieces of a tile: a warp's terms
constexpr int SEQ_PIECE = SEQ_TILE / SEQ_PIECES;

// ---------------------------------------------------------------------------
// Producers over the plain 2^n layout.
// ---------------------------------------------------------------------------
template <class T>
struct ProdHalf {        // amplitudes with bit t == outcome, ascending
    const cplx<T> *amps;
    unsigned t;
    uint64_t obit;
    __device__ __forceinline__ uint64_t index(uint64_t j) const { return insert0(j, t) | obit; }
    __device__ __forceinline__ cplx<T> amp(uint64_t j) const { return amps[index(j)]; }
    __device__ __forceinline__ T p(uint64_t j) const
    {
        const cplx<T> a = amp(j);
        return norm2_rn(a.x, a.y);
    }
};

template <class T>
struct ProdAll {         // every amplitude, ascending
    const cplx<T> *amps;
    __device__ __forceinline__ uint64_t index(uint64_t j) const { return j; }
    __device__ __forceinline__ cplx<T> amp(uint64_t j) const { return amps[j]; }
    __device__ __forceinline__ T p(uint64_t j) const
    {
        const cplx<T> a = amp(j);
        return norm2_rn(a.x, a.y);
    }
};

// |a|^2 of N amplitudes a thread, RN(RN(x x) + RN(y y)); all lanes call it.
// complex128: the FP64 pipe alone would take three operations a term.  A warp
// whose parts are all easy (lean.cuh) takes squares on the integer pipes, about
// 20 instructions each.  k_seq_steps leaves the pipe the other square and the
// sum (BOTH false): with the sum alone its ALU pipe, which counts the grid steps,
// is the fuller one.  Over all 2^28 amplitudes of a dense state 1649 us with no
// square on the integer pipes, 1306 with both, 1205 with one; over half of them
// 653 with one, 735 for the three lowest qubits.  The walk, one CTA
// that waits for its terms, leaves the sum alone: 138 -> 126 us at 20 qubits.
template <bool BOTH, int N>
__device__ __forceinline__ void norms(const float2 (&a)[N], float (&p)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++) p[i] = norm2_rn(a[i].x, a[i].y);
}
template <bool BOTH, int N>
__device__ __forceinline__ void norms(const double2 (&a)[N], double (&p)[N])
{
    auto bits = [](double v) { return uint64_t(__double_as_longlong(v)); };
    auto square = [&](double v) { return __longlong_as_double((long long)emu::lean_square(bits(v))); };
    bool easy = true;
#pragma unroll
    for (int i = 0; i < N; i++) easy &= emu::easy_square(bits(a[i].x)) & (!BOTH || emu::easy_square(bits(a[i].y)));
    if (__all_sync(0xffffffffu, easy)) {
#pragma unroll
        for (int i = 0; i < N; i++)
            p[i] = __dadd_rn(square(a[i].x), BOTH ? square(a[i].y) : __dmul_rn(a[i].y, a[i].y));
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) p[i] = norm2_rn(a[i].x, a[i].y);
    }
}

// ---------------------------------------------------------------------------
// Scans of transducers.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum_d(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ Tx shfl_up_tx(const Tx &t, unsigned off)
{
    Tx r;
    r.d[0] = __shfl_up_sync(0xffffffffu, (unsigned long long)t.d[0], off);
    r.d[1] = __shfl_up_sync(0xffffffffu, (unsigned long long)t.d[1], off);
    return r;
}

__device__ __forceinline__ Tx warp_scan_incl(Tx x)
{
    // inclusive ordered scan: lane l holds lanes 0..l composed in order
    const unsigned lane = threadIdx.x & 31;
    for (unsigned off = 1; off < 32; off <<= 1) {
        const Tx y = shfl_up_tx(x, off);
        if (lane >= off) x = tx_then(y, x);
    }
    return x;
}

__device__ __forceinline__ uint64_t warp_min_u(uint64_t v)
{
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t w = __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
        v = w < v ? w : v;
    }
    return v;
}

// ---------------------------------------------------------------------------
// 1. Estimates.  One warp per tile adds 64 terms, in four pieces spread over
// the tile: a guess of a binade needs no more, and the pass reads 1/64 of the
// state.  k_seq_whole adds all of them, one CTA per tile, for the few tiles of
// a small state.
// ---------------------------------------------------------------------------
template <class Prod>
__global__ void __launch_bounds__(SEQ_TPB) k_seq_estimate(Prod pr, uint64_t count, uint64_t ntiles,
                                                          double *__restrict__ out)
{
    const unsigned lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (SEQ_TPB / 32);
    for (uint64_t b = uint64_t(blockIdx.x) * (SEQ_TPB / 32) + (threadIdx.x >> 5); b < ntiles; b += warps) {
        const uint64_t base = b * SEQ_TILE;
        double acc = 0, n = 0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint64_t j = base + (lane >> 3) * (SEQ_TILE / 4) + (lane & 7) + 8 * k;
            if (j < count) {
                acc += double(pr.p(j));
                n += 1;
            }
        }
        acc = warp_sum_d(acc);
        n = warp_sum_d(n);
        const double all = double(count - base < uint64_t(SEQ_TILE) ? count - base : uint64_t(SEQ_TILE));
        if (lane == 0) out[b] = n > 0 ? acc * (all / n) : 0.0;
    }
}

template <class Prod>
__global__ void __launch_bounds__(SEQ_TPB) k_seq_whole(Prod pr, uint64_t count, double *__restrict__ out)
{
    __shared__ double red[SEQ_TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = uint64_t(blockIdx.x) * SEQ_TILE;
    double acc = 0;
#pragma unroll
    for (int k = 0; k < SEQ_PER; k++) {
        const uint64_t j = base + uint64_t(k * SEQ_TPB + int(threadIdx.x));
        if (j < count) acc += double(pr.p(j));
    }
    acc = warp_sum_d(acc);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = red[0];
        for (int w = 1; w < SEQ_TPB / 32; w++) v += red[w];
        out[blockIdx.x] = v;
    }
}

// ---------------------------------------------------------------------------
// 2, 4. Guesses.  One CTA; thread t takes consecutive tiles.  With `redo`
// the guesses are compared with the ones the steps were counted for, and the
// tiles that differ are listed (redo[0]: their number).
// ---------------------------------------------------------------------------
constexpr int SEQ_GUESS_TPB = 1024;

enum SeqFlag : uint8_t {
    SEQ_BIG = 1,       // a term or the tile's steps do not fit the binade
    SEQ_NONE = 2,      // no guess of a normal binade
    SEQ_ZERO = 4       // every term is zero
};

template <class A>
__global__ void __launch_bounds__(SEQ_GUESS_TPB) k_seq_guess(const double *__restrict__ est, uint64_t ntiles,
                                                            int16_t *__restrict__ guess, uint32_t *__restrict__ redo,
                                                            const uint8_t *__restrict__ flags)
{
    __shared__ double wsum[32];
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t per = (ntiles + SEQ_GUESS_TPB - 1) / SEQ_GUESS_TPB, b0 = tid * per;
    const uint64_t b1 = b0 + per < ntiles ? b0 + per : ntiles;
    double mine = 0;
    for (uint64_t b = b0; b < b1; b++) mine += est[b];
    double incl = mine;
    for (unsigned off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    double run = incl - mine;
    for (unsigned w = 0; w < warp; w++) run += wsum[w];
    if (run < 0) run = 0;                              // rounding of incl - mine
    for (uint64_t b = b0; b < b1; b++) {
        const double end = run + est[b];
        const int16_t g = int16_t(binade<A>(A(run > 0 ? run : end)));
        if (redo) {
            if (!(flags[b] & SEQ_ZERO) && g != guess[b]) {
                guess[b] = g;
                redo[1 + atomicAdd(redo, 1u)] = uint32_t(b);
            }
        } else {
            guess[b] = g;
        }
        run = end;
    }
}

// ---------------------------------------------------------------------------
// 3. Steps.  Warp w of a tile's CTA takes the piece of 512 consecutive terms
// from 512 w on, its lanes 32 consecutive ones at a time, so every load of a
// warp is coalesced.  Step counts just add up, in any order, unless a term is
// a rounding tie; a warp with a tie does its piece again, composing the terms
// in order.
//
// Bound by the FP64 pipe (a square and the sum a term, 69% busy) and the ALU
// pipe (the other square, the step counts, 68%) together, at 0.46 of HBM.  Two
// passes over the state with the sums of the first in FP64, a host step between
// them and 32-way conflicts in shared memory took 2.3 ms for the probability of
// one qubit of 28; this and the redone tiles take 0.7.
// ---------------------------------------------------------------------------
// Packs a term's grid steps with its tie bit (bit 63); steps never reach
// 2^62 without also raising `big`.
constexpr uint64_t TIE_BIT = uint64_t(1) << 63;

// Grid steps of p >= 0 in binade e as grid_steps<A>, packed: the common case
// (a normal term below the binade, by a shift of less than 64) first.
template <class A, class P>
__device__ __forceinline__ uint64_t packed_steps(P p, int e, bool &big)
{
    using TP = fp_traits<P>;
    const auto b = to_bits(p);
    const int ef = int(b >> TP::MANT);                        // p is not negative
    const int sh = (e - fp_traits<A>::MANT) - (ef - TP::BIAS - TP::MANT);
    if (ef > 0 && ef < TP::EXPMASK && sh >= 1 + TP::MANT - fp_traits<A>::MANT && sh >= 1 && sh < 64) {
        const uint64_t m = uint64_t(b & ((typename TP::bits_t(1) << TP::MANT) - 1)) | (uint64_t(1) << TP::MANT);
        const uint64_t t = m >> (sh - 1);                     // the steps and the half
        const bool tie = (t & 1) && (m << (65 - sh)) == 0 && (sh > 1);
        if (sh == 1) return (t >> 1) | ((t & 1) ? TIE_BIT : 0);
        return tie ? (t >> 1) | TIE_BIT : (t + 1) >> 1;
    }
    bool tie, bg;
    uint64_t v = grid_steps<A>(p, e, tie, bg);
    if (bg) {
        big = true;
        return 0;
    }
    return v | (tie ? TIE_BIT : 0);
}

// A thread's steps, added up: quick() takes a term by 32-bit shifts of its
// significand -- twice the steps and a half bit, whose rounding (up, away from
// a tie) is the half bit again, so a sum of truncated doubles and a count of
// half bits hold the total -- and declines what needs more: terms of more
// than half the binade, suspected ties, and every term of a very low binade.
// 25 instructions a term, with packed_steps alone 60.
template <class A, class P>
struct StepSum {
    uint64_t sum = 0, ties = 0;
    bool big = false;
    __device__ __forceinline__ explicit StepSum(int e_) : e(e_) {}
    __device__ __forceinline__ void add(P p)
    {
        const uint64_t v = packed_steps<A>(p, e, big);
        sum += v & ~TIE_BIT;
        ties |= v;
    }
    __device__ __forceinline__ uint64_t total() const { return sum; }
    int e;
};
template <>
struct StepSum<double, double> {
    uint64_t sum = 0, twice = 0, ties = 0;
    uint32_t odd = 0;
    bool big = false;
    __device__ __forceinline__ explicit StepSum(int e_) : e(e_) {}
    __device__ __forceinline__ void add(double p)
    {
        const uint32_t hi = uint32_t(__double2hiint(p)), lo = uint32_t(__double2loint(p));
        const int k = (e + 1022) - int(hi >> 20);              // bits below the half bit
        const uint32_t mh = (hi & 0x000FFFFFu) | 0x00100000u;
        const bool far = k >= 32;
        const uint32_t tl = far ? __funnelshift_rc(mh, 0u, unsigned(k) - 32u) : __funnelshift_rc(lo, mh, unsigned(k));
        const uint32_t th = __funnelshift_rc(mh, 0u, unsigned(k));
        const uint32_t below = far ? lo : lo << (32 - k);
        // with e + 1022 >= 56 a zero or a subnormal term shifts out whatever
        // its hidden bit, and with k < 1 (an infinity or NaN too) it declines
        if (k < 1 || e + 1022 < 56 || ((tl & 1u) && below == 0)) {
            const uint64_t v = packed_steps<double>(p, e, big);
            sum += v & ~TIE_BIT;
            ties |= v;
        } else {
            twice += (uint64_t(th) << 32) | tl;
            odd += tl & 1u;
        }
    }
    __device__ __forceinline__ uint64_t total() const { return sum + ((twice + odd) >> 1); }
    int e;
};

template <class Prod, class A>
__global__ void __launch_bounds__(SEQ_TPB, 4) k_seq_steps(Prod pr, uint64_t count, uint64_t ntiles,
                                                          const int16_t *__restrict__ guess,
                                                          const uint32_t *__restrict__ redo,
                                                          uint64_t *__restrict__ steps, uint64_t *__restrict__ pieces,
                                                          uint8_t *__restrict__ flags, double *__restrict__ est)
{
    // of this tile and the one before, which thread 0 may still be at
    __shared__ Tx ptxs[2][SEQ_PIECES];
    __shared__ unsigned seen[2][SEQ_PIECES];
    __shared__ double psum[SEQ_PIECES];
    constexpr uint64_t CAP = uint64_t(1) << (fp_traits<A>::MANT + 1);
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t todo = redo ? redo[0] : ntiles;
    unsigned turn = 0;
    for (uint64_t i = blockIdx.x; i < todo; i += gridDim.x, turn ^= 1) {
        Tx *const ptx = ptxs[turn];
        const uint64_t b = redo ? redo[1 + i] : i;
        const uint64_t first = b * SEQ_TILE + warp * SEQ_PIECE + lane;
        const int e = guess[b];
        const bool any = e >= fp_traits<A>::EMIN;
        using P = decltype(pr.p(uint64_t(0)));
        StepSum<A, P> mine(e);
        bool nonzero = false;
#pragma unroll 1
        for (int k = 0; k < SEQ_PIECE; k += 32 * SEQ_AHEAD) {
            decltype(pr.amp(uint64_t(0))) a[SEQ_AHEAD];
            P p[SEQ_AHEAD];
#pragma unroll
            for (int u = 0; u < SEQ_AHEAD; u++) {
                a[u].x = a[u].y = P(0);
                if (first + k + 32 * u < count) a[u] = pr.amp(first + k + 32 * u);
            }
            norms<false>(a, p);
#pragma unroll
            for (int u = 0; u < SEQ_AHEAD; u++) {
                nonzero |= to_bits(p[u]) != 0;
                if (any) mine.add(p[u]);
            }
        }
        bool big = mine.big;
        uint64_t sum = mine.total();
        const uint64_t ties = mine.ties;
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, (unsigned long long)sum, o);
        Tx t{{sum, sum}};
        if (__any_sync(0xffffffffu, (ties & TIE_BIT) != 0)) {
            t = tx_identity();
            for (int k = 0; k < SEQ_PIECE; k += 32) {
                uint64_t v = 0;
                if (first + k < count) v = packed_steps<A>(pr.p(first + k), e, big);
                const Tx inc = warp_scan_incl(tx_term(v & ~TIE_BIT, (v & TIE_BIT) != 0));
                Tx all;
                all.d[0] = __shfl_sync(0xffffffffu, (unsigned long long)inc.d[0], 31);
                all.d[1] = __shfl_sync(0xffffffffu, (unsigned long long)inc.d[1], 31);
                t = tx_then(t, all);
            }
        }
        const unsigned saw = (__any_sync(0xffffffffu, big) ? 1u : 0u) | (__any_sync(0xffffffffu, nonzero) ? 2u : 0u);
        if (lane == 0) {
            ptx[warp] = t;
            seen[turn][warp] = saw;
            if (pieces) {
                pieces[2 * (b * SEQ_PIECES + warp)] = t.d[0];
                pieces[2 * (b * SEQ_PIECES + warp) + 1] = t.d[1];
            }
        }
        __syncthreads();
        unsigned all = 0;
#pragma unroll
        for (int w = 0; w < SEQ_PIECES; w++) all |= seen[turn][w];
        const bool big_all = (all & 1u) != 0, some = (all & 2u) != 0;
        const bool lost = big_all || (!any && some);
        if (lost) {                                       // the steps do not give the tile's sum
            double acc = 0;
            for (int k = 0; k < SEQ_PIECE; k += 32)
                if (first + k < count) acc += double(pr.p(first + k));
            acc = warp_sum_d(acc);
            if (lane == 0) psum[warp] = acc;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            Tx tot = ptx[0];
            for (int w = 1; w < SEQ_PIECES; w++) tot = tx_then(tot, ptx[w]);
            uint8_t fl = 0;
            if (!some) fl = SEQ_ZERO;
            else if (!any) fl = SEQ_NONE;
            else if (big_all || tot.d[0] >= CAP || tot.d[1] >= CAP) fl = SEQ_BIG;
            steps[2 * b] = tot.d[0];
            steps[2 * b + 1] = tot.d[1];
            flags[b] = fl;
            double sum_est = 0;
            if (lost)
                for (int w = 0; w < SEQ_PIECES; w++) sum_est += psum[w];
            else if (some) sum_est = ldexp(double(tot.d[0]), e - fp_traits<A>::MANT);
            est[b] = sum_est;
        }
    }
}

// ---------------------------------------------------------------------------
// 5. The walk.
// ---------------------------------------------------------------------------
// Threads: fewer leave the SM idle in the terms, more wait longer in the scans
// (ten probabilities of a 28-qubit state walk in 4.5 / 3.4 / 3.1 / 3.7 ms with
// 128 / 256 / 512 / 1024).
constexpr int SEQ_WALK_TPB = 512, SEQ_WALK_WARPS = SEQ_WALK_TPB / 32;
constexpr int SEQ_RUN = 16;                            // tiles a thread takes per round
constexpr int SEQ_TERMS = SEQ_TILE / SEQ_WALK_TPB;     // most terms a thread takes of a tile per round
constexpr uint64_t SEQ_END = ~uint64_t(0);

template <class A> __device__ __forceinline__ A from_bits(uint64_t b);
template <> __device__ __forceinline__ double from_bits<double>(uint64_t b) { return __longlong_as_double((long long)b); }
template <> __device__ __forceinline__ float from_bits<float>(uint64_t b) { return __uint_as_float(uint32_t(b)); }

template <class A> struct rn_add;
template <> struct rn_add<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
};
template <> struct rn_add<float> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
};

// Grid positions from this one up lie outside any binade; counts are capped
// here, so that the sums of a scan over the CTA stay below 2^62.
constexpr uint64_t SEQ_CAP = uint64_t(1) << 54;

struct WalkShared {
    uint64_t count[2][SEQ_WALK_WARPS];
    Tx tx[SEQ_WALK_WARPS];
    uint64_t least[SEQ_WALK_WARPS];
    uint64_t pos, at;        // where a round ended: the position (or sum) and the next item
};

__device__ __forceinline__ uint64_t block_min(uint64_t v, WalkShared &sh)
{
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_min_u(v);
    __syncthreads();
    if (lane == 0) sh.least[warp] = v;
    __syncthreads();
    return warp_min_u(sh.least[lane % SEQ_WALK_WARPS]);
}

// The effect on a sum of what the threads before this one add: this thread's
// steps when the sum is even or odd (they differ only with a rounding tie).
// Returns the grid position before this thread's part, given the round's
// start m0.  One barrier when no thread has a tie; `turn` alternates.
__device__ __forceinline__ uint64_t scan_from(uint64_t m0, Tx mine, WalkShared &sh, unsigned turn)
{
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = mine.d[0] < SEQ_CAP ? mine.d[0] : SEQ_CAP;
    const uint64_t own = incl;
    for (unsigned off = 1; off < 32; off <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, (unsigned long long)incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) sh.count[turn][warp] = incl < SEQ_CAP ? incl : SEQ_CAP;
    if (!__syncthreads_or(mine.d[0] != mine.d[1])) {
        uint64_t before = 0;
#pragma unroll
        for (unsigned w = 0; w < SEQ_WALK_WARPS; w++)
            if (w < warp) before += sh.count[turn][w];
        return m0 + before + (incl - own);
    }
    const Tx inc = warp_scan_incl(mine);
    if (lane == 31) sh.tx[warp] = inc;
    __syncthreads();
    Tx before = tx_identity(), excl = shfl_up_tx(inc, 1);
    for (unsigned w = 0; w < warp; w++) before = tx_then(before, sh.tx[w]);
    __syncthreads();                                   // sh.tx is read
    if (lane == 0) excl = tx_identity();
    excl = tx_then(before, excl);
    return m0 + excl.d[m0 & 1];
}

template <class A>
__device__ __forceinline__ bool finite_sum(A s)
{
    return int((to_bits(s) >> fp_traits<A>::MANT) & fp_traits<A>::EXPMASK) != fp_traits<A>::EXPMASK;
}

// The exact running sum after the terms tm[0..valid) from `s`; every thread
// returns it.  A sum that starts at zero leaves a binade every time the number
// of terms doubles: its rounds span four times the terms before them.
// Where term i lies in shared memory: a gap after every 16, so that threads
// with 16 (or 8) consecutive terms each read from different banks.
__device__ __forceinline__ unsigned term_slot(unsigned i) { return i + (i >> 4); }

template <class A, class P>
__device__ A walk_terms(const P *tm, unsigned valid, A s, WalkShared &sh, unsigned &turn)
{
    constexpr uint64_t LIM = uint64_t(1) << (fp_traits<A>::MANT + 1);
    const unsigned tid = threadIdx.x;
    const bool small = s == A(0);
    unsigned i = 0, per = small ? 1 : SEQ_TERMS;
    while (i < valid) {
        const int e = binade(s);
        if (!finite_sum(s)) {
            // an infinity or a NaN only changes at a NaN
            bool nan = false;
            for (unsigned r = i + tid; r < valid; r += SEQ_WALK_TPB) nan |= tm[term_slot(r)] != tm[term_slot(r)];
            if (__syncthreads_or(nan)) s = A(s + A(NAN));
            return s;
        }
        if (e < fp_traits<A>::EMIN) {
            if (s == A(0)) {
                // skip to the first nonzero term
                uint64_t nz = SEQ_END;
                for (unsigned r = i + tid; r < valid && nz == SEQ_END; r += SEQ_WALK_TPB)
                    if (to_bits(tm[term_slot(r)]) != 0) nz = r;
                nz = block_min(nz, sh);
                if (nz == SEQ_END) return s;
                i = unsigned(nz);
            }
            s = rn_add<A>::add(s, A(tm[term_slot(i)]));       // zero or subnormal: one term
            i++;
            continue;
        }
        // a round of terms [i, end) in binade e; the thread in whose terms the
        // sum leaves the binade walks them and adds the one that does
        const unsigned most = i + SEQ_WALK_TPB * per, end = most < valid ? most : valid;
        const unsigned lo = i + tid * per, hi = lo + per < end ? lo + per : end;
        StepSum<A, P> steps(e);
        for (unsigned r = lo; r < hi; r++) steps.add(tm[term_slot(r)]);
        const uint64_t ties = steps.ties;
        Tx mine;
        mine.d[0] = steps.big ? SEQ_CAP : steps.total();     // one term leaves the binade by itself
        mine.d[1] = mine.d[0];
        auto term = [&](unsigned r) {
            bool big = false;
            const uint64_t v = packed_steps<A>(tm[term_slot(r)], e, big);
            return big ? Tx{{SEQ_CAP, SEQ_CAP}} : tx_term(v & ~TIE_BIT, (v & TIE_BIT) != 0);
        };
        if (ties & TIE_BIT) {
            mine = tx_identity();
            for (unsigned r = lo; r < hi; r++) mine = tx_then(mine, term(r));
        }
        uint64_t pos = scan_from(grid_pos(s), mine, sh, turn);
        turn ^= 1;
        if (lo < hi && pos < LIM) {
            if (pos + mine.d[pos & 1] >= LIM) {    // the one thread where it crosses
                unsigned r = lo;
                for (; r + 1 < hi; r++) {
                    const uint64_t step = term(r).d[pos & 1];
                    if (pos + step >= LIM) break;
                    pos += step;
                }
                sh.pos = to_bits(rn_add<A>::add(grid_at<A>(pos, e), A(tm[term_slot(r)])));
                sh.at = r + 1;
            } else if (hi == end) {
                sh.pos = to_bits(grid_at<A>(pos + mine.d[pos & 1], e));
                sh.at = end;
            }
        }
        __syncthreads();
        s = from_bits<A>(sh.pos);
        i = unsigned(sh.at);
        if (small) per = i < 64 ? 1 : i >= 64 * SEQ_TERMS ? SEQ_TERMS : (i + 63) / 64;
    }
    return s;
}

// starts (or null): the running sum before each tile; inside[b]: the binade
// it stays in throughout tile b, or EMIN - 1 where the tile was walked term
// by term.  out: the total.
template <class Prod, class P, class A>
__global__ void __launch_bounds__(SEQ_WALK_TPB) k_seq_walk(Prod pr, uint64_t count, uint64_t ntiles,
                                                           const int16_t *__restrict__ guess,
                                                           const uint64_t *__restrict__ steps,
                                                           const uint8_t *__restrict__ flags,
                                                           double *__restrict__ starts, int16_t *__restrict__ inside,
                                                           double *__restrict__ out)
{
    __shared__ P tm[SEQ_TILE + SEQ_TILE / 16];
    __shared__ WalkShared sh;
    constexpr uint64_t LIM = uint64_t(1) << (fp_traits<A>::MANT + 1);
    const unsigned tid = threadIdx.x;
    A s = A(0);
    uint64_t t = 0;
    unsigned turn = 0;
    while (t < ntiles) {
        const int e = binade(s);
        uint64_t bad = t;
        if (s == A(0)) {
            // to the first tile that is not all zeros
            const uint64_t most = t + uint64_t(SEQ_WALK_TPB) * SEQ_RUN;
            const uint64_t end = most < ntiles ? most : ntiles;
            uint64_t some = SEQ_END;
            for (uint64_t b = t + tid; b < end; b += SEQ_WALK_TPB)
                if (some == SEQ_END && !(flags[b] & SEQ_ZERO)) some = b;
            some = block_min(some, sh);
            const uint64_t stop = some == SEQ_END ? end : some;
            if (starts)
                for (uint64_t b = t + tid; b < stop; b += SEQ_WALK_TPB) {
                    starts[b] = 0.0;
                    inside[b] = int16_t(fp_traits<A>::EMIN - 1);
                }
            t = stop;
            bad = some;
        } else if (e >= fp_traits<A>::EMIN && finite_sum(s)) {
            // a round of tiles [t, end) that stay in binade e
            const uint64_t most = t + uint64_t(SEQ_WALK_TPB) * SEQ_RUN;
            const uint64_t end = most < ntiles ? most : ntiles;
            const int per = int((end - t + SEQ_WALK_TPB - 1) / SEQ_WALK_TPB);
            const uint64_t b0 = t + uint64_t(tid) * unsigned(per);
            auto effect = [&](uint64_t b) {
                const uint8_t f = flags[b];
                const int g = guess[b];
                const ulonglong2 d = reinterpret_cast<const ulonglong2 *>(steps)[b];
                if (f & SEQ_ZERO) return tx_identity();
                if (f || g != e) return Tx{{LIM, LIM}};      // stops here
                return Tx{{d.x < LIM ? d.x : LIM, d.y < LIM ? d.y : LIM}};
            };
            Tx mine = tx_identity();
            bool parity = false;
#pragma unroll 4
            for (int r = 0; r < per; r++)
                if (b0 + r < end) {
                    const Tx x = effect(b0 + r);
                    parity |= x.d[0] != x.d[1];
                    mine.d[0] += x.d[0];
                }
            mine.d[1] = mine.d[0];
            if (parity) {
                mine = tx_identity();
                for (int r = 0; r < per; r++)
                    if (b0 + r < end) mine = tx_then(mine, effect(b0 + r));
            }
            uint64_t pos = scan_from(grid_pos(s), mine, sh, turn);
            turn ^= 1;
            if (b0 < end && pos < LIM) {
                const uint64_t last = b0 + unsigned(per) < end ? b0 + unsigned(per) : end;
                const uint64_t fin = pos + mine.d[pos & 1];
                if (fin >= LIM || starts) {                  // the tile the round stops before; the starts
                    uint64_t b = b0;
                    for (; b < last; b++) {
                        const uint64_t d = effect(b).d[pos & 1];
                        if (pos + d >= LIM) break;
                        if (starts) {
                            starts[b] = double(grid_at<A>(pos, e));
                            inside[b] = int16_t(e);
                        }
                        pos += d;
                    }
                    if (b < last || last == end) {
                        sh.pos = pos;
                        sh.at = b;
                    }
                } else if (last == end) {
                    sh.pos = fin;
                    sh.at = end;
                }
            }
            __syncthreads();
            s = grid_at<A>(sh.pos, e);
            t = sh.at;
            bad = t < end ? t : SEQ_END;
        }
        if (bad == SEQ_END) continue;
        // tile t term by term
        if (starts && tid == 0) {
            starts[t] = double(s);
            inside[t] = int16_t(fp_traits<A>::EMIN - 1);
        }
        if (!(flags[t] & SEQ_ZERO)) {
            const uint64_t base = t * SEQ_TILE;
            const unsigned valid = unsigned(count - base < uint64_t(SEQ_TILE) ? count - base : uint64_t(SEQ_TILE));
            __syncthreads();
            decltype(pr.amp(uint64_t(0))) a[SEQ_TERMS];
            P v[SEQ_TERMS];
#pragma unroll
            for (int r = 0; r < SEQ_TERMS; r++) {
                const unsigned i = unsigned(r) * SEQ_WALK_TPB + tid;
                a[r].x = a[r].y = P(0);
                if (i < valid) a[r] = pr.amp(base + i);
            }
            norms<true>(a, v);
#pragma unroll
            for (int r = 0; r < SEQ_TERMS; r++) tm[term_slot(unsigned(r) * SEQ_WALK_TPB + tid)] = v[r];
            __syncthreads();
            s = walk_terms<A, P>(tm, valid, s, sh, turn);
            __syncthreads();
        }
        t++;
    }
    if (tid == 0) *out = double(s);
}

// ---------------------------------------------------------------------------
// 6. Shots: one warp per uniform.
// ---------------------------------------------------------------------------
template <class Prod, class A>
__global__ void __launch_bounds__(SEQ_TPB) k_seq_shots(Prod pr, uint64_t count, uint64_t ntiles,
                                                       const double *__restrict__ starts,
                                                       const int16_t *__restrict__ inside,
                                                       const uint64_t *__restrict__ pieces,
                                                       const double *__restrict__ total, const double *__restrict__ u,
                                                       uint32_t nshots, int strict, uint64_t *__restrict__ out)
{
    const uint32_t shot = blockIdx.x * (SEQ_TPB / 32) + (threadIdx.x >> 5);
    const unsigned lane = threadIdx.x & 31;
    if (shot >= nshots) return;
    const double x = u[shot];
    auto reaches = [strict, x](double v) { return strict ? v > x : v >= x; };
    if (!reaches(*total)) {                                // past the total (:167, :258)
        if (lane == 0) out[shot] = strict ? ~uint64_t(0) : 0;
        return;
    }
    if (reaches(0.0)) {                                    // the first partial sum does
        if (lane == 0) out[shot] = pr.index(0);
        return;
    }
    // the first tile whose end reaches x
    uint64_t lo = 0, hi = ntiles - 1;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (reaches(starts[mid + 1])) hi = mid;
        else lo = mid + 1;
    }
    const uint64_t b = lo;
    A s = A(starts[b]);
    uint64_t i = b * SEQ_TILE;
    const uint64_t tile_end = i + SEQ_TILE < count ? i + SEQ_TILE : count;
    // first grid position of binade e whose value reaches x
    auto target = [strict, x](int e) {
        const A xa = A(x);
        uint64_t g;
        if (sizeof(A) == 8 || double(xa) == x) g = grid_ceil<A>(xa, e);
        else g = grid_ceil<A>(double(xa) < x ? A(__uint_as_float(__float_as_uint(float(xa)) + 1u)) : xa, e);
        if (strict && ldexp(double(g), e - fp_traits<A>::MANT) == x) g++;
        return g;
    };
    const int e0 = inside[b];
    if (e0 >= fp_traits<A>::EMIN) {
        // to the piece that reaches it
        const uint64_t tgt = target(e0);
        uint64_t pos = grid_pos(s);
        for (int w = 0; w + 1 < SEQ_PIECES; w++) {
            const ulonglong2 d = reinterpret_cast<const ulonglong2 *>(pieces)[b * SEQ_PIECES + w];
            const uint64_t next = pos + ((pos & 1) ? d.y : d.x);
            if (next >= tgt) break;
            pos = next;
            i += SEQ_PIECE;
        }
        s = grid_at<A>(pos, e0);
    }
    // the terms from i on, a round of 32 x SEQ_PER at a time
    uint64_t found = tile_end - 1;
    while (i < tile_end) {
        const int e = binade(s);
        if (e < fp_traits<A>::EMIN || !finite_sum(s)) {
            if (s == A(0)) {
                // past zero terms, 32 at a time (a zero sum reaches no x > 0)
                const uint64_t j = i + lane;
                const unsigned nz = __ballot_sync(0xffffffffu, j < tile_end && to_bits(pr.p(j)) != 0);
                if (!nz) {
                    i += 32;
                    continue;
                }
                i += unsigned(__ffs(nz) - 1);
            }
            s = rn_add<A>::add(s, A(pr.p(i)));
            if (reaches(double(s))) {
                found = i;
                break;
            }
            i++;
            continue;
        }
        const uint64_t end = i + 32 * SEQ_PER < tile_end ? i + 32 * SEQ_PER : tile_end;
        const uint64_t base = i + uint64_t(lane) * SEQ_PER;
        const unsigned len = base < end ? unsigned(end - base < uint64_t(SEQ_PER) ? end - base : SEQ_PER) : 0u;
        auto run = [&pr, base](unsigned r) { return pr.p(base + r); };
        bool big = false;
        const Tx incl = warp_scan_incl(run_effect<A>(run, len, e, big));
        Tx excl = shfl_up_tx(incl, 1);
        if (lane == 0) excl = tx_identity();
        const uint64_t m0 = grid_pos(s);
        const uint64_t pos0 = m0 + excl.d[m0 & 1];
        uint64_t pos = pos0;
        const unsigned walked = run_walk<A>(run, len, e, pos);
        const uint64_t bad = warp_min_u(walked < len ? base + walked : SEQ_END);
        const uint64_t stop = bad == SEQ_END ? end : bad;
        const uint64_t tgt = target(e);
        const unsigned hit = __ballot_sync(0xffffffffu, len && base < stop && pos >= tgt);
        if (hit) {
            const unsigned L = unsigned(__ffs(hit) - 1);
            uint64_t j = 0;
            if (lane == L) j = base + run_find<A>(run, len, e, pos0, tgt);
            found = __shfl_sync(0xffffffffu, (unsigned long long)j, L);
            break;
        }
        const uint64_t last = bad == SEQ_END ? end - 1 : stop;
        const uint64_t pend = __shfl_sync(0xffffffffu, (unsigned long long)pos, unsigned((last - i) / SEQ_PER));
        s = grid_at<A>(pend, e);
        i = stop;
        if (bad != SEQ_END) {
            s = rn_add<A>::add(s, A(pr.p(i)));             // the term that leaves the binade
            if (reaches(double(s))) {
                found = i;
                break;
            }
            i++;
        }
    }
    if (lane == 0) out[shot] = pr.index(found);
}

// ---------------------------------------------------------------------------
// Host side: working storage carved from one block, and the launches.
// ---------------------------------------------------------------------------
struct SeqScratch {
    double *total;          // 8 bytes
    double *est;
    uint64_t *steps;        // two per tile
    int16_t *guess;
    uint8_t *flags;
    uint32_t *redo;         // a count, then up to one entry per tile
    double *starts;         // sampling only, from here on
    int16_t *inside;
    uint64_t *pieces;
    size_t bytes;
    static size_t align(size_t x) { return (x + 255) & ~size_t(255); }
    static SeqScratch carve(void *base, uint64_t ntiles, bool sampling)
    {
        SeqScratch s{};
        char *p = static_cast<char *>(base);
        size_t off = 0;
        auto take = [&](auto *&q, size_t n) {
            q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(p + off);
            off += align(n);
        };
        take(s.total, 8);
        take(s.est, ntiles * 8);
        take(s.steps, ntiles * 16);
        take(s.guess, ntiles * 2);
        take(s.flags, ntiles);
        take(s.redo, (ntiles + 1) * 4);
        if (sampling) {
            take(s.starts, ntiles * 8);
            take(s.inside, ntiles * 2);
            take(s.pieces, ntiles * SEQ_PIECES * 16);
        }
        s.bytes = off;
        return s;
    }
};

// The sum of producer `pr` over `count` elements, left in sc.total.
template <class Prod, class P, class A>
int seq_launch(cudaStream_t str, uint64_t *launches, const SeqScratch &sc, const Prod &pr, uint64_t count)
{
    const uint64_t ntiles = (count + SEQ_TILE - 1) / SEQ_TILE;
    // few tiles: their sums are read whole, and need no second look
    const bool whole = ntiles <= 512;
    const unsigned wgrid = unsigned(std::min<uint64_t>((ntiles + SEQ_TPB / 32 - 1) / (SEQ_TPB / 32), sm_count() * 8));
    const unsigned grid = unsigned(std::min<uint64_t>(ntiles, uint64_t(sm_count()) * 6));
    if (whole) k_seq_whole<Prod><<<unsigned(ntiles), SEQ_TPB, 0, str>>>(pr, count, sc.est);
    else k_seq_estimate<Prod><<<wgrid, SEQ_TPB, 0, str>>>(pr, count, ntiles, sc.est);
    k_seq_guess<A><<<1, SEQ_GUESS_TPB, 0, str>>>(sc.est, ntiles, sc.guess, nullptr, nullptr);
    k_seq_steps<Prod, A><<<grid, SEQ_TPB, 0, str>>>(pr, count, ntiles, sc.guess, nullptr, sc.steps, sc.pieces, sc.flags,
                                                    sc.est);
    *launches += 4;
    if (!whole) {
        QSLC_CUDA(cudaMemsetAsync(sc.redo, 0, 4, str));
        k_seq_guess<A><<<1, SEQ_GUESS_TPB, 0, str>>>(sc.est, ntiles, sc.guess, sc.redo, sc.flags);
        k_seq_steps<Prod, A><<<grid, SEQ_TPB, 0, str>>>(pr, count, ntiles, sc.guess, sc.redo, sc.steps, sc.pieces,
                                                        sc.flags, sc.est);
        *launches += 2;
    }
    k_seq_walk<Prod, P, A><<<1, SEQ_WALK_TPB, 0, str>>>(pr, count, ntiles, sc.guess, sc.steps, sc.flags, sc.starts,
                                                        sc.inside, sc.total);
    QSLC_CUDA(cudaGetLastError());
    return QSLC_OK;
}

// The sum over a handle's growable scratch, on the host.
template <class Prod, class P, class A>
int seq_total(qslc_state *s, const Prod &pr, uint64_t count, double *out)
{
    const uint64_t ntiles = (count + SEQ_TILE - 1) / SEQ_TILE;
    int rc = s->scratch.ensure(SeqScratch::carve(nullptr, ntiles, false).bytes);
    if (!rc) rc = ensure_pinned(s, 8);
    if (rc) return rc;
    const SeqScratch sc = SeqScratch::carve(s->scratch.ptr, ntiles, false);
    rc = seq_launch<Prod, P, A>(s->stream, &s->launches, sc, pr, count);
    if (rc) return rc;
    QSLC_CUDA(cudaMemcpyAsync(s->host_pinned, sc.total, 8, cudaMemcpyDeviceToHost, s->stream));
    QSLC_CUDA(cudaStreamSynchronize(s->stream));
    *out = *static_cast<double *>(s->host_pinned);
    return QSLC_OK;
}

// Sampling: for each uniform, the basis index of the element whose partial
// sum is the first to reach it, into out[0..n) in the order of u.
// strict (sampleAll2, measure.cpp:237-267): the first element whose
// partial sum exceeds u; a uniform at or above the total lands nowhere and
// is reported as ~0.  Otherwise (sampleAll): the first partial sum >= u,
// and 0 above the total.
template <class Prod, class P, class A>
int seq_sample(qslc_state *s, const Prod &pr, uint64_t count, const double *u, uint64_t n, uint64_t *out,
               bool strict = false)
{
    const uint64_t ntiles = (count + SEQ_TILE - 1) / SEQ_TILE;
    int rc = s->scratch.ensure(SeqScratch::carve(nullptr, ntiles, true).bytes);
    if (!rc) rc = s->scratch2.ensure(2 * SeqScratch::align(n * 8));
    if (rc) return rc;
    const SeqScratch sc = SeqScratch::carve(s->scratch.ptr, ntiles, true);
    double *d_u = static_cast<double *>(s->scratch2.ptr);
    uint64_t *d_out = reinterpret_cast<uint64_t *>(static_cast<char *>(s->scratch2.ptr) + SeqScratch::align(n * 8));
    QSLC_CUDA(cudaMemcpyAsync(d_u, u, n * 8, cudaMemcpyHostToDevice, s->stream));
    rc = seq_launch<Prod, P, A>(s->stream, &s->launches, sc, pr, count);
    if (rc) return rc;
    k_seq_shots<Prod, A><<<unsigned((n + SEQ_TPB / 32 - 1) / (SEQ_TPB / 32)), SEQ_TPB, 0, s->stream>>>(
        pr, count, ntiles, sc.starts, sc.inside, sc.pieces, sc.total, d_u, uint32_t(n), strict ? 1 : 0, d_out);
    s->launches++;
    QSLC_CUDA(cudaGetLastError());
    QSLC_CUDA(cudaMemcpyAsync(out, d_out, n * 8, cudaMemcpyDeviceToHost, s->stream));
    QSLC_CUDA(cudaStreamSynchronize(s->stream));
    return QSLC_OK;
}

}  // namespace qslc
