// batch.cu -- the batching form: thousands of small circuits in one
// persistent launch, replayed from a CUDA graph.
//
// Each instance is a hardware-efficient ansatz on n qubits: L layers of
// rotateY on every qubit, rotateZ on every qubit, then controlNot(q, q+1)
// for q = 0..n-2; afterwards prob(q, 0) and prob(q, 1) for every q and a
// sampleAll draw per uniform.  The per-instance result is the one qsl's
// Default backend gives for the same calls (gates.cpp, measure.cpp), bit
// for bit: every amplitude sees the reference's operations in the
// reference's order with its rounding, the probabilities are sequential
// sums in index order, and the sampling CDF is the sequential double sum
// merged against the instance's sorted uniforms (the first index whose
// running sum reaches a uniform is its outcome, as drawSample's search
// returns, measure.cpp:164-188).
//
// The graph holds four kernels.  k_batch runs the circuits and leaves every
// instance's |a|^2 terms in global memory; k_batch_probs64 (or 32) and k_batch_cdf, side
// by side, turn them into the probabilities (chains of dependent adds, one
// per thread) and the shots; k_batch_sort, before k_batch, sorts each
// instance's uniforms for the CDF walk.
//
// Schedule of k_batch: persistent clusters of CTAs pull instances, largest
// first, from an atomic counter.  A state of at most one tile (2^k amplitudes
// of shared memory) lives in the shared memory of one CTA for its whole
// circuit, and each CTA of a cluster takes its own.  A larger state lives in
// two buffers of the cluster's slot in a global arena and takes two passes
// per layer instead of one per gate, whose tiles the CTAs of the cluster
// share:
//   pass 1  tiles of 2^k consecutive amplitudes: rotateY on qubits 0..k-1;
//   pass 2  tiles that vary the high n-k qubits and the lowest 2k-n ones:
//           rotateY on qubits k..n-1, then rotateZ on every qubit (each
//           rotateZ touches one amplitude at a time, so all n of them apply
//           per amplitude, in order), then the whole controlNot ladder as
//           one permutation into the other buffer -- or, after the last
//           layer, the |a|^2 terms in its order.
// The ladder maps basis index x to y with y_i = x_0 ^ ... ^ x_i (each
// controlNot(q, q+1) flips bit q+1 when bit q of the running index is set).
//
// The tile size, threads per CTA and CTAs per SM are picked by measuring
// the candidates on the caller's own batch (qslc_batch_autotune).
#include "gatemath.cuh"
#include "replay.cuh"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <thread>
#include <vector>

namespace qslc {
namespace {

constexpr int MAX_Q = 26;

struct InstDesc {
    uint32_t n, L;
    uint64_t coef;      // offset of its coefficients: L*n*4 values (cy, sy, cz, sz)
    uint64_t probs;     // offset of its 2n probabilities
    uint64_t shots;     // offset of its shots and uniforms
    uint64_t norms;     // offset of its 2^n |a|^2 terms
};

struct BatchArgs {
    const InstDesc *inst;
    const uint32_t *order;      // large instances, then the ones of at most a tile
    uint32_t ninst, nlarge;
    unsigned *counter;
    unsigned *pick;             // two words per cluster: the position it works on
    const void *coef;
    double *probs;
    const double *u;            // the uniforms, in the caller's order
    double *usorted;
    uint32_t *perm;             // where each sorted uniform came from
    uint64_t *shots;            // in the caller's order
    uint32_t nshots;
    void *norms;                // every instance's |a|^2 terms, in index order
    const uint32_t *size_order; // instances by qubit count, largest first
    void *arena;
    uint64_t slot_amps;         // amplitudes per arena buffer (two buffers per cluster)
    unsigned tile_log2;         // k: the shared-memory tile holds 2^k amplitudes
};

// Indices of at most MAX_Q bits.
__host__ __device__ __forceinline__ uint32_t ladder(uint32_t x)
{   // y_i = x_0 ^ ... ^ x_i
    x ^= x << 1;
    x ^= x << 2;
    x ^= x << 4;
    x ^= x << 8;
    x ^= x << 16;
    return x;
}

// ---- one gate's coefficients, in shared memory -------------------------------
template <class T> struct BatchCoef;
template <> struct BatchCoef<float> {
    float c, s;
};
template <> struct alignas(16) BatchCoef<double> {
    emu::LeanK lc, ls;
    SlowCoef head;
};
template <class T>
struct LayerCoefs {
    BatchCoef<T> ry[MAX_Q], rz[MAX_Q];
};

__device__ __forceinline__ BatchCoef<float> batch_coef(float c, float s) { return BatchCoef<float>{c, s}; }
__device__ __forceinline__ BatchCoef<double> batch_coef(double c, double s)
{
    return BatchCoef<double>{emu::make_lean_gate(c), emu::make_lean_gate(s),
                             SlowCoef{c, s, emu::make_mulk(c), emu::make_mulk(s)}};
}

template <class T>
__device__ __forceinline__ void stage_layer(LayerCoefs<T> &lc, const T *cf, uint32_t n)
{
    const unsigned tid = threadIdx.x;
    __syncthreads();                                  // the last layer's readers
    if (tid < 2 * n) {
        const uint32_t q = tid >> 1;
        const T *c = cf + 4 * q + 2 * (tid & 1);
        (tid & 1 ? lc.rz : lc.ry)[q] = batch_coef(c[0], c[1]);
    }
    __syncthreads();
}

// A thread's amplitudes in registers: 4 of 16 bytes (two rotateY per visit
// of shared memory) or 16 of 8 bytes (four).  With two of each, complex64
// was bound by shared memory and barriers: 262 ms for 4096 instances.
template <class T> constexpr int BR = sizeof(T) == 8 ? 2 : 4;

// Where local amplitude l lies in the tile (linear in l; see run.cu).
template <class T>
__device__ __forceinline__ uint32_t slot_of(uint32_t l)
{
    if constexpr (sizeof(T) == 8) return l ^ ((0x2570u >> (4 * ((l >> 3) & 3u))) & 7u);
    else return l ^ ((l >> 4) & 15u);
}

// rotateY along register bit P (gates.cpp:169-174).
template <int P>
__device__ __forceinline__ void ry_regs(double2 (&v)[4], const BatchCoef<double> &bc)
{
    Coef<double> k{};
    k.lc = bc.lc;
    k.ls = bc.ls;
    pair_either<P_RY>(v[0], v[P == 0 ? 1 : 2], k, &bc.head, nullptr);
    pair_either<P_RY>(v[P == 0 ? 2 : 1], v[3], k, &bc.head, nullptr);
}
// (a0 c - a1 s, a0 s + a1 c), with a1 (-s) for the difference; mul.f32x2
// multiplies both parts of an amplitude, rounding each on its own.  The sums
// stay scalar: the assembler fuses an add.f32x2 with the products.
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add_parts(float2 a, float2 b)
{
    return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
template <int P>
__device__ __forceinline__ void ry_regs(float2 (&v)[1 << BR<float>], const BatchCoef<float> &bc)
{
    const float2 c = make_float2(bc.c, bc.c), s = make_float2(bc.s, bc.s), m = make_float2(-bc.s, -bc.s);
#pragma unroll
    for (int i = 0; i < (1 << BR<float>) / 2; i++) {
        const int i0 = ((i >> P) << (P + 1)) | (i & ((1 << P) - 1)), i1 = i0 | (1 << P);
        const float2 a0 = v[i0], a1 = v[i1];
        v[i0] = add_parts(mul2(a0, c), mul2(a1, m));
        v[i1] = add_parts(mul2(a0, s), mul2(a1, c));
    }
}

// rotateZ on one qubit of a thread's amplitudes: where the qubit's bit is
// clear (re*c + im*s, im*c - re*s), where it is set (re*c - im*s, im*c + re*s)
// (gates.cpp:200-205).  `ones`: bit i says whether amplitude i has it set.
__device__ __forceinline__ void rz_regs(double2 (&v)[4], const BatchCoef<double> &bc, unsigned ones)
{
    Coef<double> k{};
    k.lc = bc.lc;
    k.ls = bc.ls;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t flip = ((ones >> i) & 1u) ? 0u : 0x80000000u;
        phase_flip(v[i], flip, k, &bc.head);
    }
}
__device__ __forceinline__ void rz_regs(float2 (&v)[1 << BR<float>], const BatchCoef<float> &bc, unsigned ones)
{
#pragma unroll
    for (int i = 0; i < (1 << BR<float>); i++) {
        const float s = ((ones >> i) & 1u) ? bc.s : -bc.s;
        const float re = v[i].x, im = v[i].y;
        v[i].x = __fsub_rn(__fmul_rn(re, bc.c), __fmul_rn(im, s));
        v[i].y = __fadd_rn(__fmul_rn(im, bc.c), __fmul_rn(re, s));
    }
}
// The same where all of them agree on the bit.
__device__ __forceinline__ void rz_same(float2 (&v)[1 << BR<float>], const BatchCoef<float> &bc, bool one)
{
    const float s = one ? bc.s : -bc.s;
#pragma unroll
    for (int i = 0; i < (1 << BR<float>); i++) {
        const float re = v[i].x, im = v[i].y;
        v[i].x = __fsub_rn(__fmul_rn(re, bc.c), __fmul_rn(im, s));
        v[i].y = __fadd_rn(__fmul_rn(im, bc.c), __fmul_rn(re, s));
    }
}
__device__ __forceinline__ void rz_same(double2 (&v)[4], const BatchCoef<double> &bc, bool one)
{
    rz_regs(v, bc, one ? 15u : 0u);
}

// Register bits at tile bit `lo`: thread item q's base, and amplitude i of it.
template <class T>
__device__ __forceinline__ uint32_t item_base(uint32_t q, unsigned lo)
{
    return ((q >> lo) << (lo + BR<T>)) | (q & ((1u << lo) - 1u));
}

// The byte offsets in shared memory of an item's amplitudes: slot_of is linear,
// so they are the base's XOR a combination of BR offsets that all items share.
template <class T>
struct ItemMap {
    uint32_t off[BR<T>];
    __device__ __forceinline__ explicit ItemMap(unsigned lo)
    {
#pragma unroll
        for (int b = 0; b < BR<T>; b++) off[b] = slot_of<T>(1u << (lo + b)) * uint32_t(sizeof(cplx<T>));
    }
    __device__ __forceinline__ uint32_t at(uint32_t x, int i) const
    {
#pragma unroll
        for (int b = 0; b < BR<T>; b++)
            if (i & (1 << b)) x ^= off[b];
        return x;
    }
};
template <class T>
__device__ __forceinline__ cplx<T> &tile_at(cplx<T> *sm, uint32_t byte)
{
    return *reinterpret_cast<cplx<T> *>(reinterpret_cast<unsigned char *>(sm) + byte);
}

template <class T>
__device__ __forceinline__ void load_item(cplx<T> (&v)[1 << BR<T>], cplx<T> *sm, uint32_t base, const ItemMap<T> &m)
{
    const uint32_t x = slot_of<T>(base) * uint32_t(sizeof(cplx<T>));
#pragma unroll
    for (int i = 0; i < (1 << BR<T>); i++) v[i] = tile_at<T>(sm, m.at(x, i));
}
template <class T>
__device__ __forceinline__ void store_item(cplx<T> *sm, const cplx<T> (&v)[1 << BR<T>], uint32_t base,
                                           const ItemMap<T> &m)
{
    const uint32_t x = slot_of<T>(base) * uint32_t(sizeof(cplx<T>));
#pragma unroll
    for (int i = 0; i < (1 << BR<T>); i++) tile_at<T>(sm, m.at(x, i)) = v[i];
}

// rotateY on qubits q0..q0+cnt-1, in order, on register bits r0..r0+cnt-1.
template <class T>
__device__ __forceinline__ void ry_some(cplx<T> (&v)[1 << BR<T>], const BatchCoef<T> *ry, unsigned r0, unsigned cnt)
{
    const BatchCoef<T> *c = ry - r0;
    if (r0 <= 0 && r0 + cnt > 0) ry_regs<0>(v, c[0]);
    if (r0 <= 1 && r0 + cnt > 1) ry_regs<1>(v, c[1]);
    if constexpr (BR<T> >= 3)
        if (r0 <= 2 && r0 + cnt > 2) ry_regs<2>(v, c[2]);
    if constexpr (BR<T> == 4) {
        if (r0 <= 3 && r0 + cnt > 3) ry_regs<3>(v, c[3]);
    }
}

// rotateY on qubits q0..q1-1 of the circuit, in order, on bits off..
// off + (q1 - q0) - 1 of a tile of 2^m amplitudes, up to BR of them per visit;
// `last(v, base, lo)` takes each item of the last visit in place of the
// store.  A barrier after each visit but the last.
template <class T, class Last>
__device__ __forceinline__ void ry_layer(cplx<T> *sm, unsigned m, unsigned q0, unsigned q1, unsigned off,
                                         const LayerCoefs<T> &lc, Last last)
{
    constexpr unsigned R = BR<T>;
    const uint32_t items = 1u << (m - R);
    for (unsigned q = q0; q < q1;) {
        const unsigned cnt = q1 - q < R ? q1 - q : R;
        const unsigned b = off + (q - q0);
        const unsigned lo = b + R <= m ? b : m - R;       // the register bits lo..lo+R-1 hold bits b..b+cnt-1
        const bool end = q + cnt == q1;
        const ItemMap<T> map(lo);
        for (uint32_t it = threadIdx.x; it < items; it += blockDim.x) {
            const uint32_t base = item_base<T>(it, lo);
            cplx<T> v[1 << R];
            load_item<T>(v, sm, base, map);
            ry_some<T>(v, &lc.ry[q], b - lo, cnt);
            if (end) last(v, base, lo);
            else store_item<T>(sm, v, base, map);
        }
        if (!end) __syncthreads();
        q += cnt;
    }
}

// rotateZ on qubits 0..n-1, in that order, of a thread's amplitudes: number i
// has basis index x + (i << rb).
template <class T>
__device__ __forceinline__ void rz_all(cplx<T> (&v)[1 << BR<T>], uint32_t x, unsigned rb, uint32_t n,
                                       const LayerCoefs<T> &lc)
{
    constexpr unsigned R = BR<T>;
    for (uint32_t q = 0; q < rb; q++) rz_same(v, lc.rz[q], ((x >> q) & 1) != 0);
    rz_regs(v, lc.rz[rb], 0xAAAAu);
    rz_regs(v, lc.rz[rb + 1], 0xCCCCu);
    if constexpr (R >= 3) rz_regs(v, lc.rz[rb + 2], 0xF0F0u);
    if constexpr (R >= 4) rz_regs(v, lc.rz[rb + 3], 0xFF00u);
    for (uint32_t q = rb + R; q < n; q++) rz_same(v, lc.rz[q], ((x >> q) & 1) != 0);
}

// The same where amplitude i has basis index `index(i)`.
template <class T, class Index>
__device__ __forceinline__ void rz_each(cplx<T> (&v)[1 << BR<T>], Index index, uint32_t n, const LayerCoefs<T> &lc)
{
    for (uint32_t q = 0; q < n; q++) {
        unsigned ones = 0;
        for (unsigned i = 0; i < (1u << BR<T>); i++) ones |= unsigned((index(i) >> q) & 1) << i;
        rz_regs(v, lc.rz[q], ones);
    }
}

// An instance of at least BR qubits that fits one tile: the whole circuit in
// shared memory.  Below a whole tile the ladder goes into the tile's other
// half; a state of a whole tile takes it one controlNot at a time.
template <class T>
__device__ void run_small(cplx<T> *tile, LayerCoefs<T> &lc, const InstDesc &d, const T *coef, bool halves,
                          T *__restrict__ gn)
{
    const uint32_t n = d.n, dim = 1u << n;
    const unsigned tid = threadIdx.x, nt = blockDim.x;
    cplx<T> *sm = tile, *other = tile + (halves ? dim : 0);
    for (uint32_t i = tid; i < dim; i += nt) {
        cplx<T> z;
        z.x = T(i == 0 ? 1 : 0);
        z.y = T(0);
        sm[i] = z;                                        // slot_of(0) is 0
    }
    for (uint32_t l = 0; l < d.L; l++) {
        stage_layer<T>(lc, coef + d.coef + uint64_t(l) * n * 4, n);   // also orders the fill
        ry_layer<T>(sm, n, 0, n, 0, lc, [&](cplx<T>(&v)[1 << BR<T>], uint32_t base, unsigned lo) {
            rz_all<T>(v, base, lo, n, lc);
            if (halves) {
                // the ladder is linear too
                const uint32_t y = ladder(base);
#pragma unroll
                for (int i = 0; i < (1 << BR<T>); i++)
                    other[slot_of<T>((y ^ ladder(uint32_t(i) << lo)) & (dim - 1))] = v[i];
            } else {
                store_item<T>(sm, v, base, ItemMap<T>(lo));
            }
        });
        if (halves) {
            cplx<T> *t = sm;
            sm = other;
            other = t;
            continue;                                     // stage_layer's barrier orders the stores
        }
        for (uint32_t q = 0; q + 1 < n; q++) {            // controlNot(q, q+1), gates.cpp:215-240
            __syncthreads();
            const uint32_t cb = 1u << q, tb = 2u << q;
            for (uint32_t j = tid; j < (dim >> 2); j += nt) {
                const uint32_t x1 = uint32_t(insert00(j, q, q + 1)) | cb;
                const uint32_t s1 = slot_of<T>(x1), s2 = slot_of<T>(x1 | tb);
                const cplx<T> a = sm[s1], b = sm[s2];
                sm[s1] = b;
                sm[s2] = a;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < dim; i += nt) {
        const cplx<T> a = sm[slot_of<T>(i)];
        gn[i] = norm2_rn(a.x, a.y);
    }
}

// The instances below BR qubits, which do not fill a thread's registers.
template <class T>
__device__ void run_tiny(cplx<T> *sm, const InstDesc &d, const T *coef, T *__restrict__ gn)
{
    const uint32_t n = d.n, dim = 1u << n;
    const unsigned tid = threadIdx.x;
    if (tid < dim) {
        sm[tid].x = T(tid == 0 ? 1 : 0);
        sm[tid].y = T(0);
    }
    for (uint32_t l = 0; l < d.L; l++) {
        const T *cf = coef + d.coef + uint64_t(l) * n * 4;
        for (uint32_t q = 0; q < n; q++) {
            __syncthreads();
            Coef<T> k{};
            k.c = cf[4 * q];
            k.s = cf[4 * q + 1];
            if (tid < dim / 2) {
                const uint32_t i0 = uint32_t(insert0(tid, q));
                pair_update<T, P_RY>(sm[i0], sm[i0 | (1u << q)], k);
            }
        }
        __syncthreads();
        if (tid < dim) {
            cplx<T> a = sm[tid];
            for (uint32_t q = 0; q < n; q++) {
                const T c = cf[4 * q + 2], s = cf[4 * q + 3];
                const T sg = ((tid >> q) & 1) ? s : -s;
                const T re = a.x, im = a.y;
                a.x = rn<T>::sub(rn<T>::mul(re, c), rn<T>::mul(im, sg));
                a.y = rn<T>::add(rn<T>::mul(im, c), rn<T>::mul(re, sg));
            }
            sm[(ladder(tid) & (dim - 1)) + dim] = a;
        }
        __syncthreads();
        if (tid < dim) sm[tid] = sm[tid + dim];
    }
    __syncthreads();
    if (tid < dim) gn[tid] = norm2_rn(sm[tid].x, sm[tid].y);
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// The state's buffers are written by one CTA of a cluster and read by
// another: read past the L1.
__device__ __forceinline__ double2 load_shared_state(const double2 *p) { return __ldcg(p); }
__device__ __forceinline__ float2 load_shared_state(const float2 *p) { return __ldcg(p); }

// An instance larger than a tile: two buffers in the cluster's arena slot, two
// passes per layer, tile t of a pass done by CTA t mod the cluster's size.
template <class T>
__device__ void run_large(cplx<T> *sm, LayerCoefs<T> &lc, const InstDesc &d, const T *coef, cplx<T> *buf0,
                          cplx<T> *buf1, unsigned k, unsigned rank, unsigned ctas, T *__restrict__ gn)
{
    constexpr unsigned R = BR<T>, A = 1u << R;
    const uint32_t n = d.n;
    const uint32_t dim = 1u << n, tile = 1u << k;
    const unsigned tid = threadIdx.x, nt = blockDim.x;
    const unsigned h = n - k;                 // qubits above the tile (h <= k)
    const unsigned c = k - h;                 // low qubits that pass-2 tiles keep whole
    const uint32_t cmask = (1u << c) - 1;
    cplx<T> *src = buf0, *dst = buf1;
    for (uint32_t i = rank * nt + tid; i < dim; i += ctas * nt) {
        cplx<T> z;
        z.x = T(i == 0 ? 1 : 0);
        z.y = T(0);
        src[i] = z;
    }
    if (d.L == 0) {
        for (uint32_t i = rank * nt + tid; i < dim; i += ctas * nt) gn[i] = T(i == 0 ? 1 : 0);
        return;
    }
    for (uint32_t l = 0; l < d.L; l++) {
        const bool final_layer = l + 1 == d.L;
        stage_layer<T>(lc, coef + d.coef + uint64_t(l) * n * 4, n);
        cluster_sync();                       // the buffer the last pass wrote
        // pass 1: rotateY on qubits 0..k-1, tile by tile, in place
        for (uint32_t t = rank; t < (1u << h); t += ctas) {
            cplx<T> *g = src + (uint64_t(t) << k);
            for (uint32_t i0 = tid; i0 < tile; i0 += 4 * nt) {
                cplx<T> v[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i0 + u * nt < tile) v[u] = load_shared_state(g + i0 + u * nt);
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i0 + u * nt < tile) sm[slot_of<T>(i0 + u * nt)] = v[u];
            }
            __syncthreads();
            ry_layer<T>(sm, k, 0, k, 0, lc, [&](cplx<T>(&v)[A], uint32_t base, unsigned lo) {
#pragma unroll
                for (unsigned i = 0; i < A; i++) g[base | (i << lo)] = v[i];
            });
            __syncthreads();
        }
        cluster_sync();
        // pass 2: tile t fixes bits c..k-1 of the index to t; local index
        // l = (high bits << c) | (low c bits)
        for (uint32_t t = rank; t < (1u << h); t += ctas) {
            const uint32_t mid = t << c;
            for (uint32_t i0 = tid; i0 < tile; i0 += 4 * nt) {
                cplx<T> v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t i = i0 + u * nt;
                    if (i < tile) v[u] = load_shared_state(src + (((i >> c) << k) | mid | (i & cmask)));
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i0 + u * nt < tile) sm[slot_of<T>(i0 + u * nt)] = v[u];
            }
            __syncthreads();
            ry_layer<T>(sm, k, k, n, c, lc, [&](cplx<T>(&v)[A], uint32_t base, unsigned lo) {
                // the index of amplitude 0; the register bits may reach below
                // bit c when few qubits lie above the tile
                auto index = [&](uint32_t loc) { return ((loc >> c) << k) | mid | (loc & cmask); };
                if (lo >= c) rz_all<T>(v, index(base), lo - c + k, n, lc);
                else rz_each<T>(v, [&](unsigned i) { return index(base | (i << lo)); }, n, lc);
                const uint32_t y0 = ladder(index(base));
#pragma unroll
                for (unsigned i = 0; i < A; i++) {
                    const uint32_t y = (y0 ^ ladder(((i << lo) >> c << k) | ((i << lo) & cmask))) & (dim - 1);
                    if (final_layer) gn[y] = norm2_rn(v[i].x, v[i].y);
                    else dst[y] = v[i];
                }
            });
            __syncthreads();
        }
        cplx<T> *tmp = src;
        src = dst;
        dst = tmp;
    }
}

// THREADS: the most threads of a CTA; 512 for a lone one of 512 threads an SM,
// which then has 128 registers each.
template <class T, int THREADS>
__global__ void __launch_bounds__(THREADS) k_batch(BatchArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ LayerCoefs<T> lc;
    cplx<T> *sm = reinterpret_cast<cplx<T> *>(smem_raw);
    const T *coef = static_cast<const T *>(a.coef);
    T *norms = static_cast<T *>(a.norms);
    const unsigned rank = cluster_rank(), ctas = cluster_size(), id = blockIdx.x / ctas;
    cplx<T> *slot = static_cast<cplx<T> *>(a.arena) + uint64_t(id) * 2 * a.slot_amps;
    const uint32_t nsmall = a.ninst - a.nlarge, all = a.nlarge + (nsmall + ctas - 1) / ctas;
    for (unsigned round = 0;; round ^= 1) {
        // one pick for the cluster; the word of the round before last is free
        if (rank == 0 && threadIdx.x == 0) {
            a.pick[2 * id + round] = atomicAdd(a.counter, 1u);
            __threadfence();
        }
        cluster_sync();
        const uint32_t w = __ldcg(a.pick + 2 * id + round);
        if (w >= all) break;
        const uint32_t at = w < a.nlarge ? w : a.nlarge + (w - a.nlarge) * ctas + rank;
        if (at >= a.ninst) continue;
        const InstDesc d = a.inst[a.order[at]];
        T *gn = norms + d.norms;
        if (w < a.nlarge) run_large<T>(sm, lc, d, coef, slot, slot + a.slot_amps, a.tile_log2, rank, ctas, gn);
        else if (d.n < unsigned(BR<T>)) run_tiny<T>(sm, d, coef, gn);
        else run_small<T>(sm, lc, d, coef, d.n < a.tile_log2, gn);
        __syncthreads();
    }
}

// The probabilities, after k_batch: prob(q, o) is the sequential Fp sum, in
// index order, of the terms with bit q == o (measure.cpp:126-147), a chain of
// dependent adds with one thread per sum and two warps per instance.
//
// complex128: an FP64 add holds its quarter of the SM for 64 clocks whatever
// the active lanes, so what counts is the steps of a warp, and every thread
// goes at its own next term.  The terms come straight from L2, PROB_AHEAD of
// them loaded while as many are added; the threads' addresses lie apart, and
// 16-byte loads keep the load unit behind the adds.  On 1024 instances of up
// to 20 qubits 40 ms; passed through shared
// memory, where the lanes of high qubits idle while those of low ones add, 64.
constexpr unsigned PROB_THREADS = 128, PROB_AHEAD = 8;

__global__ void __launch_bounds__(PROB_THREADS) k_batch_probs64(BatchArgs a)
{
    const uint32_t w = 2 * blockIdx.x + (threadIdx.x >> 6);
    if (w >= a.ninst) return;
    const InstDesc d = a.inst[a.size_order[w]];
    const double *__restrict__ gn = static_cast<const double *>(a.norms) + d.norms;
    const uint32_t sum = threadIdx.x & 63u, q = sum >> 1, o = sum & 1;
    if (sum >= 2 * d.n) return;
    const uint32_t half = 1u << (d.n - 1), ob = o << q, low = (1u << q) - 1u;
    const uint32_t ahead = half < PROB_AHEAD ? half : PROB_AHEAD;
    // an instance's terms begin at a multiple of 4 of them, and a run of 8 from
    // qubit 3 up at a multiple of 8
    const bool wide = q >= 3 && half >= PROB_AHEAD && (d.norms & 1) == 0;
    auto load = [&](double (&v)[PROB_AHEAD], uint32_t j) {
        if (wide) {
            const double2 *r = reinterpret_cast<const double2 *>(gn + ((((j & ~low) << 1) | (j & low)) | ob));
#pragma unroll
            for (uint32_t i = 0; i < PROB_AHEAD / 2; i++) {
                const double2 t = r[i];
                v[2 * i] = t.x;
                v[2 * i + 1] = t.y;
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < PROB_AHEAD; i++)
                if (i < ahead) {
                    const uint32_t x = j + i;
                    v[i] = gn[(((x & ~low) << 1) | (x & low)) | ob];
                }
        }
    };
    double p = 0.0, cur[PROB_AHEAD], nxt[PROB_AHEAD];
    load(cur, 0);
    for (uint32_t j = 0; j < half; j += ahead) {
        if (j + ahead < half) load(nxt, j + ahead);
#pragma unroll
        for (uint32_t i = 0; i < PROB_AHEAD; i++)
            if (i < ahead) p = __dadd_rn(p, cur[i]);
#pragma unroll
        for (uint32_t i = 0; i < PROB_AHEAD; i++) cur[i] = nxt[i];
    }
    a.probs[d.probs + sum] = p;
}

// complex64: an FP32 add is quick, and the terms pass through shared memory a
// tile of 2^k at a time.  Warp 0 adds the sums of qubits below k (half of each
// tile), warp 1 those of the others (a whole tile or none); the slots spread
// the lanes' addresses, which differ in one bit, over the banks.  20 ms for 4096
// instances.
constexpr unsigned PROBF_LOG2 = 11;

__global__ void __launch_bounds__(64) k_batch_probs32(BatchArgs a)
{
    __shared__ float tm[1u << PROBF_LOG2];
    auto slot = [](uint32_t x) { return x ^ ((x >> 5) & 31u) ^ (3u * ((x >> 10) & 1u)); };
    const InstDesc d = a.inst[a.size_order[blockIdx.x]];
    const float *__restrict__ gn = static_cast<const float *>(a.norms) + d.norms;
    const uint32_t n = d.n, k = n < PROBF_LOG2 ? n : PROBF_LOG2, size = 1u << k;
    const uint32_t lane = threadIdx.x & 31u, q = (threadIdx.x < 32 ? 0u : k) + (lane >> 1), o = lane & 1;
    const bool sums = threadIdx.x < 32 ? q < k : q < n;
    const uint32_t low = (1u << q) - 1u, ob = o << q;
    float p = 0.f;
    for (uint32_t c = 0; c < (1u << (n - k)); c++) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < size; i += 64) tm[slot(i)] = gn[(uint64_t(c) << k) + i];
        __syncthreads();
        if (!sums) continue;
        if (threadIdx.x < 32) {
#pragma unroll 8
            for (uint32_t j = 0; j < (size >> 1); j++)
                p = __fadd_rn(p, tm[slot((((j & ~low) << 1) | (j & low)) | ob)]);
        } else if (((c >> (q - k)) & 1) == o) {
#pragma unroll 8
            for (uint32_t i = 0; i < size; i++) p = __fadd_rn(p, tm[slot(i)]);
        }
    }
    if (sums) a.probs[d.probs + 2 * q + o] = double(p);
}

// Each instance's uniforms in ascending order, by counting for each the ones
// below it (equal ones in the caller's order); uniforms pass through shared
// memory a piece at a time.  The work grows with the square of nshots, so
// larger counts are sorted on the host: 4096 instances of 1024 shots take
// under 1 ms here and took 13 ms on 16 host cores.
constexpr unsigned SORT_THREADS = 256, SORT_PIECE = 2048, SORT_MAX = 4096;

template <class T>
__global__ void __launch_bounds__(SORT_THREADS) k_batch_sort(BatchArgs a)
{
    __shared__ double piece[SORT_PIECE];
    const uint32_t ns = a.nshots, id = blockIdx.x;
    const double *u = a.u + uint64_t(id) * ns;
    for (uint32_t i0 = 0; i0 < ns; i0 += SORT_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        const double mine = i < ns ? u[i] : 0.0;
        const long long key = __double_as_longlong(mine);          // uniforms are not negative
        uint32_t below = 0;
        for (uint32_t p0 = 0; p0 < ns; p0 += SORT_PIECE) {
            const uint32_t len = ns - p0 < SORT_PIECE ? ns - p0 : SORT_PIECE;
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < len; j += SORT_THREADS) piece[j] = u[p0 + j];
            __syncthreads();
            for (uint32_t j = 0; j < len; j++) {
                const long long other = __double_as_longlong(piece[j]);
                below += (other < key) | ((other == key) & (p0 + j < i));
            }
        }
        if (i < ns) {
            a.usorted[uint64_t(id) * ns + below] = double(T(mine));   // the reference draws Fp uniforms
            a.perm[uint64_t(id) * ns + below] = i;
        }
    }
}

// The sampling CDFs, after k_batch, one CTA per instance.  A uniform's outcome
// is the first index whose running double sum of |a|^2 terms reaches it, index
// 0 when none does (measure.cpp:60-78, :164-188).  The running sum s is exact
// at all times:
//   - while s is normal, in binade e, a round of CDF_THREADS x CDF_RUN terms
//     runs in parallel: each thread takes CDF_RUN consecutive terms, a scan of
//     their grid-step transducers (replay.cuh) over the CTA gives every thread
//     the grid position where its run starts, and each walks its run; the
//     round stops before the first term whose sum would leave the binade (or
//     that is too big for it), which is then added on its own with one FP64
//     add;
//   - while s is zero, zero terms are skipped a CTA's width at a time, and
//     while it is subnormal, terms are added one at a time.
// After every term, all uniforms the sum has reached take that term's index,
// so the outcomes are the sequential merge's; within a round each thread
// looks up a uniform of its own.  A round's latency bounds the walk of the
// largest instance: rounds of 4096 terms instead of a warp's 512 took the
// kernel from 18 to 5 ms on 1024 instances of up to 20 qubits.
constexpr unsigned CDF_RUN = 16, CDF_THREADS = 256, CDF_WARPS = CDF_THREADS / 32;
constexpr uint64_t CDF_NONE = ~uint64_t(0);

// The test u <= run, for u in [0, 1) and run >= 0: the bit patterns of
// non-negative doubles order like their values, so integer compares keep it
// off the FP64 pipe.
__device__ __forceinline__ bool cdf_reached(double u, double run)
{
    return __double_as_longlong(u) <= __double_as_longlong(run);
}

__device__ __forceinline__ Tx shfl_up_tx(const Tx &t, unsigned off)
{
    Tx r;
    r.d[0] = __shfl_up_sync(0xFFFFFFFFu, (unsigned long long)t.d[0], off);
    r.d[1] = __shfl_up_sync(0xFFFFFFFFu, (unsigned long long)t.d[1], off);
    return r;
}

template <class T>
__global__ void __launch_bounds__(CDF_THREADS) k_batch_cdf(BatchArgs a)
{
    __shared__ Tx warp_tx[CDF_WARPS];
    __shared__ uint64_t warp_bad[CDF_WARPS], first[CDF_THREADS], after[CDF_THREADS];
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t id = a.size_order[blockIdx.x];
    const InstDesc d = a.inst[id];
    const T *__restrict__ nr = static_cast<const T *>(a.norms) + d.norms;
    const double *__restrict__ u = a.usorted + uint64_t(id) * a.nshots;
    const uint32_t *__restrict__ perm = a.perm + uint64_t(id) * a.nshots;
    uint64_t *__restrict__ out = a.shots + d.shots;
    const uint64_t dim = uint64_t(1) << d.n;
    const uint32_t ns = a.nshots;
    uint32_t k = 0;                                       // next uniform
    double s = 0.0;                                       // the sum of terms 0..i-1
    uint64_t i = 0;                                       // next term
    // the least of the threads' values (all of them call it)
    auto least = [&](uint64_t v) {
        for (unsigned off = 16; off; off >>= 1) {
            const uint64_t o = __shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)v, off);
            v = o < v ? o : v;
        }
        __syncthreads();
        if (lane == 0) warp_bad[warp] = v;
        __syncthreads();
        v = warp_bad[0];
        for (unsigned w = 1; w < CDF_WARPS; w++) v = warp_bad[w] < v ? warp_bad[w] : v;
        return v;
    };
    // the uniforms from k on that `take(u)` accepts (a leading part of them)
    // get outcomes, a CTA's width at a time
    auto consume = [&](auto take, auto outcome) {
        for (;;) {
            const uint32_t j = k + tid;
            const bool t = j < ns && take(u[j]);
            if (t) out[perm[j]] = outcome(u[j]);
            const unsigned c = unsigned(__syncthreads_count(t));
            k += c;
            if (c < CDF_THREADS) break;
        }
    };
    auto reached = [&](double x) { return cdf_reached(x, s); };
    while (i < dim && k < ns) {
        const int e = binade(s);
        if (e < fp_traits<double>::EMIN) {
            if (__double_as_longlong(s) == 0) {
                // zero so far: skip to the first nonzero term
                const uint64_t j = i + tid;
                const uint64_t nz = least(j < dim && to_bits(nr[j]) != 0 ? j : CDF_NONE);
                consume(reached, [&](double) { return i; });   // u == 0 is reached at term i
                if (nz == CDF_NONE) {
                    i = i + CDF_THREADS < dim ? i + CDF_THREADS : dim;
                    continue;
                }
                i = nz;
            }
            s = __dadd_rn(s, double(nr[i]));              // subnormal (or zero) sum: one term
            consume(reached, [&](double) { return i; });
            i++;
            continue;
        }
        // a round of terms [i, end) in binade e
        const uint64_t m0 = grid_pos(s);
        const uint64_t end = i + CDF_THREADS * CDF_RUN < dim ? i + CDF_THREADS * CDF_RUN : dim;
        const uint64_t base = i + uint64_t(tid) * CDF_RUN;
        const unsigned len = base < end ? unsigned(end - base < CDF_RUN ? end - base : CDF_RUN) : 0u;
        auto run = [nr, base](unsigned r) { return nr[base + r]; };
        bool big = false;
        Tx incl = run_effect<double>(run, len, e, big);
        for (unsigned off = 1; off < 32; off <<= 1) {
            const Tx o = shfl_up_tx(incl, off);
            if (lane >= off) incl = tx_then(o, incl);
        }
        Tx excl = shfl_up_tx(incl, 1);
        if (lane == 0) excl = tx_identity();
        __syncthreads();                                  // the last round's readers
        if (lane == 31) warp_tx[warp] = incl;
        __syncthreads();
        Tx before = tx_identity();
        for (unsigned w = 0; w < warp; w++) before = tx_then(before, warp_tx[w]);
        excl = tx_then(before, excl);
        const uint64_t pos0 = m0 + excl.d[m0 & 1];        // grid position before this thread's run
        uint64_t pos = pos0;
        const unsigned walked = run_walk<double>(run, len, e, pos);
        const uint64_t bad = least(walked < len ? base + walked : CDF_NONE);
        const uint64_t stop = bad == CDF_NONE ? end : bad;
        // the position after term stop - 1: where the thread holding `stop`
        // stopped, or where the one holding the round's last term ended
        const uint64_t last = bad == CDF_NONE ? end - 1 : stop;
        const unsigned holder = unsigned((last - i) / CDF_RUN);
        first[tid] = pos0;
        after[tid] = pos;
        __syncthreads();
        const uint64_t pend = after[holder];
        // uniforms reached inside [i, stop): the first run, and in it the
        // first term, whose position reaches the uniform's grid target
        const uint64_t i0 = i;
        const unsigned live = holder + (last < stop || last > i0 + uint64_t(holder) * CDF_RUN ? 1u : 0u);
        consume([&](double x) { return live && grid_ceil<double>(x, e) <= pend; },
                [&](double x) {
                    const uint64_t tgt = grid_ceil<double>(x, e);
                    unsigned lo = 0, hi = live - 1;       // the first run with after >= tgt
                    while (lo < hi) {
                        const unsigned mid = (lo + hi) >> 1;
                        if (after[mid] >= tgt) hi = mid;
                        else lo = mid + 1;
                    }
                    const uint64_t b = i0 + uint64_t(lo) * CDF_RUN;
                    const unsigned ln = unsigned(end - b < CDF_RUN ? end - b : CDF_RUN);
                    auto other = [nr, b](unsigned r) { return nr[b + r]; };
                    return b + run_find<double>(other, ln, e, first[lo], tgt);
                });
        s = grid_at<double>(pend, e);
        i = stop;
        if (bad != CDF_NONE) {
            s = __dadd_rn(s, double(nr[i]));              // the term that leaves the binade
            consume(reached, [&](double) { return i; });
            i++;
        }
    }
    for (uint32_t j = k + tid; j < ns; j += CDF_THREADS) out[perm[j]] = 0;   // above the total: index 0
}

}  // namespace
}  // namespace qslc

using namespace qslc;

// One launch shape of the persistent kernel.
struct BatchShape {
    unsigned threads = 1024;
    unsigned tile_log2 = 13;
    unsigned ctas_per_sm = 1;
};

struct qslc_batch {
    int dtype = QSLC_C128;
    uint32_t ninst = 0, nshots = 0, nmax = 0;
    std::vector<InstDesc> inst;
    std::vector<uint32_t> order, size_order;   // by cost and by qubit count, largest first
    std::vector<unsigned char> coef;           // the last call's coefficients
    uint64_t ncoef = 0, nprobs = 0, nshot_total = 0, nnorm_total = 0;
    cudaStream_t stream = nullptr, side = nullptr;
    cudaEvent_t forked = nullptr, joined = nullptr;
    void *d_inst = nullptr, *d_order = nullptr, *d_counter = nullptr, *d_coef = nullptr;
    void *d_probs = nullptr, *d_u = nullptr, *d_shots = nullptr, *d_arena = nullptr;
    void *d_norms = nullptr, *d_size_order = nullptr, *d_pick = nullptr, *d_usorted = nullptr, *d_perm = nullptr;
    uint64_t arena_bytes = 0, slot_amps = 0;
    BatchShape shape;
    unsigned grid = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t runs = 0;
};

namespace {

// The arena holds two buffers of 2^nmax amplitudes per cluster; beyond this
// many bytes the grid shrinks instead.
constexpr uint64_t ARENA_CAP = uint64_t(64) << 30;

size_t amp_bytes(int dtype) { return dtype == QSLC_C128 ? 16 : 8; }

void drop_graph(qslc_batch *b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

void batch_free(qslc_batch *b)
{
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    drop_graph(b);
    for (void *p : {b->d_inst, b->d_order, b->d_counter, b->d_coef, b->d_probs, b->d_u, b->d_shots,
                    b->d_arena, b->d_norms, b->d_size_order, b->d_pick, b->d_usorted, b->d_perm})
        if (p) cudaFree(p);
    if (b->forked) cudaEventDestroy(b->forked);
    if (b->joined) cudaEventDestroy(b->joined);
    if (b->side) cudaStreamDestroy(b->side);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

// Whether a shape can run this batch: the tile must fit a CTA's shared
// memory and cover at least half of the largest instance's qubits.
bool shape_fits(const qslc_batch *b, const BatchShape &s)
{
    const size_t tile = (size_t(1) << s.tile_log2) * amp_bytes(b->dtype);
    if (tile * s.ctas_per_sm + 16 * 1024 * s.ctas_per_sm > 224 * 1024) return false;
    if (s.threads * s.ctas_per_sm > 1024) return false;   // registers: 64 K per SM, up to 64 a thread
    if (b->nmax > 2 * s.tile_log2) return false;
    return true;
}

// CTAs per cluster of k_batch: enough that the largest instance does not hold
// the batch up.  The estimate, in amplitudes x layers x qubits per SM: the work
// shared by the SMs that clusters of this size can fill, and half the longest
// instance, split over a cluster, for the uneven end.
unsigned cluster_of(const qslc_batch *b, const BatchShape &s, size_t smem, const void *kernel, unsigned *clusters)
{
    double work = 0, longest = 0, alone = 0;
    for (const InstDesc &d : b->inst) {
        const double c = std::ldexp(double(std::max(d.L, 1u)) * d.n, int(d.n));
        work += c;
        (d.n > s.tile_log2 ? longest : alone) = std::max(d.n > s.tile_log2 ? longest : alone, c);
    }
    unsigned best = 1;
    double least = -1;
    for (unsigned g = 1; g <= 8; g *= 2) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim = {g, 1, 1};
        cfg.gridDim = dim3(g);
        cfg.blockDim = dim3(s.threads);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) {
            cudaGetLastError();
            continue;
        }
        const double t = work / (double(fit) * g) + 0.5 * std::max(longest / g, alone);
        if (least < 0 || t < least) {
            least = t;
            best = g;
            *clusters = unsigned(fit);
        }
    }
    if (least < 0) *clusters = sm_count();
    return best;
}

// (Re)capture the graph for shape `s`: clusters, arena size, kernel attributes.
template <class T>
int capture(qslc_batch *b, const BatchShape &s)
{
    drop_graph(b);
    const size_t ab = amp_bytes(b->dtype);
    const size_t smem = (size_t(1) << s.tile_log2) * ab;
    auto *kernel = s.threads <= 512 && s.ctas_per_sm == 1 ? k_batch<T, 512> : k_batch<T, 1024>;
    QSLC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    b->slot_amps = b->nmax > s.tile_log2 ? (uint64_t(1) << b->nmax) : 0;
    unsigned clusters = 1;
    const unsigned ctas = cluster_of(b, s, smem, reinterpret_cast<const void *>(kernel), &clusters);
    if (b->slot_amps) {
        const uint64_t slot = 2 * b->slot_amps * ab;
        clusters = unsigned(std::min<uint64_t>(clusters, std::max<uint64_t>(1, ARENA_CAP / slot)));
    }
    // large instances first, each by all CTAs of a cluster; then the others
    std::vector<uint32_t> order;
    for (uint32_t i : b->order)
        if (b->inst[i].n > s.tile_log2) order.push_back(i);
    const uint32_t nlarge = uint32_t(order.size());
    for (uint32_t i : b->order)
        if (b->inst[i].n <= s.tile_log2) order.push_back(i);
    clusters = std::min<unsigned>(clusters, nlarge + (b->ninst - nlarge + ctas - 1) / ctas);
    const uint64_t need = uint64_t(clusters) * 2 * b->slot_amps * ab;
    if (need > b->arena_bytes) {
        if (b->d_arena) cudaFree(b->d_arena);
        b->d_arena = nullptr;
        b->arena_bytes = 0;
        if (cudaMalloc(&b->d_arena, std::max<uint64_t>(need, 16)) != cudaSuccess) {
            cudaGetLastError();
            return fail(QSLC_EOOM, "out of device memory for the batch arena");
        }
        b->arena_bytes = need;
    }
    // after the last run, which reads it, and before the next
    QSLC_CUDA(cudaMemcpyAsync(b->d_order, order.data(), b->ninst * 4, cudaMemcpyHostToDevice, b->stream));
    QSLC_CUDA(cudaStreamSynchronize(b->stream));
    BatchArgs a;
    a.inst = static_cast<const InstDesc *>(b->d_inst);
    a.order = static_cast<const uint32_t *>(b->d_order);
    a.ninst = b->ninst;
    a.nlarge = nlarge;
    a.counter = static_cast<unsigned *>(b->d_counter);
    a.pick = static_cast<unsigned *>(b->d_pick);
    a.coef = b->d_coef;
    a.probs = static_cast<double *>(b->d_probs);
    a.u = static_cast<const double *>(b->d_u);
    a.usorted = static_cast<double *>(b->d_usorted);
    a.perm = static_cast<uint32_t *>(b->d_perm);
    a.shots = static_cast<uint64_t *>(b->d_shots);
    a.nshots = b->nshots;
    a.norms = b->d_norms;
    a.size_order = static_cast<const uint32_t *>(b->d_size_order);
    a.arena = b->d_arena;
    a.slot_amps = b->slot_amps;
    a.tile_log2 = s.tile_log2;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {ctas, 1, 1};
    cfg.gridDim = dim3(clusters * ctas);
    cfg.blockDim = dim3(s.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    QSLC_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(b->d_counter, 0, sizeof(unsigned), b->stream);
    if (b->nshots && b->nshots <= SORT_MAX) k_batch_sort<T><<<b->ninst, SORT_THREADS, 0, b->stream>>>(a);
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    cudaEventRecord(b->forked, b->stream);
    cudaStreamWaitEvent(b->side, b->forked, 0);
    if constexpr (sizeof(T) == 8) k_batch_probs64<<<(b->ninst + 1) / 2, PROB_THREADS, 0, b->side>>>(a);
    else k_batch_probs32<<<b->ninst, 64, 0, b->side>>>(a);
    if (b->nshots) k_batch_cdf<T><<<b->ninst, CDF_THREADS, 0, b->stream>>>(a);
    cudaEventRecord(b->joined, b->side);
    cudaStreamWaitEvent(b->stream, b->joined, 0);
    cudaGraph_t g = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(b->stream, &g);
    if (e != cudaSuccess || e2 != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return cuda_fail(e != cudaSuccess ? e : e2, "capture of the batch");
    }
    b->graph = g;
    QSLC_CUDA(cudaGraphInstantiate(&b->exec, g, 0));
    b->shape = s;
    b->grid = clusters * ctas;
    return QSLC_OK;
}

int capture_any(qslc_batch *b, const BatchShape &s)
{
    return b->dtype == QSLC_C128 ? capture<double>(b, s) : capture<float>(b, s);
}

// f(i) for every i in [0, n) on the host's cores: instance i goes to thread
// i mod T, so instances of every size spread over the threads.  Each f(i)
// touches only instance i's data.
template <class F>
void host_parallel(uint32_t n, F &&f)
{
    unsigned nt = std::thread::hardware_concurrency();
    nt = std::min<unsigned>(std::max<unsigned>(nt, 1u), 32u);
    if (nt < 2 || n < 256) {
        for (uint32_t i = 0; i < n; i++) f(i);
        return;
    }
    std::vector<std::thread> pool;
    pool.reserve(nt);
    for (unsigned t = 0; t < nt; t++)
        pool.emplace_back([&f, n, nt, t] {
            for (uint32_t i = t; i < n; i += nt) f(i);
        });
    for (auto &th : pool) th.join();
}

// Coefficients exactly as the reference computes them (gates.cpp:154-155,
// :185-186: Fp cos/sin of Fp(angle)/2), uploaded with the uniforms.  More
// than SORT_MAX uniforms an instance are sorted here (in Fp, as the reference
// draws them), with the permutation that brings the shots back.
template <class T>
int upload_inputs(qslc_batch *b, const double *angles, const double *u)
{
    b->coef.resize(b->ncoef * sizeof(T));
    T *coef = reinterpret_cast<T *>(b->coef.data());
    // instance i's angles start at 2 x (its coefficients' offset) / 4
    host_parallel(b->ninst, [&](uint32_t i) {
        const InstDesc &d = b->inst[i];
        const double *ai = angles + d.coef / 2;
        for (uint64_t k = 0; k < uint64_t(d.L) * d.n; k++) {
            const T ry = T(ai[2 * k]), rz = T(ai[2 * k + 1]);
            T *c = coef + d.coef + 4 * k;
            c[0] = T(std::cos(ry / 2));
            c[1] = T(std::sin(ry / 2));
            c[2] = T(std::cos(rz / 2));
            c[3] = T(std::sin(rz / 2));
        }
    });
    QSLC_CUDA(cudaMemcpyAsync(b->d_coef, coef, b->ncoef * sizeof(T), cudaMemcpyHostToDevice, b->stream));
    const uint32_t ns = b->nshots;
    if (ns <= SORT_MAX) {
        if (ns) QSLC_CUDA(cudaMemcpyAsync(b->d_u, u, b->nshot_total * 8, cudaMemcpyHostToDevice, b->stream));
        QSLC_CUDA(cudaStreamSynchronize(b->stream));
        return QSLC_OK;
    }
    std::vector<double> us(b->nshot_total);
    std::vector<uint32_t> perm(b->nshot_total);
    host_parallel(b->ninst, [&](uint32_t i) {
        uint32_t *pm = perm.data() + uint64_t(i) * ns;
        const double *ui = u + uint64_t(i) * ns;
        std::iota(pm, pm + ns, 0u);
        std::sort(pm, pm + ns, [&](uint32_t x, uint32_t y) { return ui[x] < ui[y]; });
        for (uint32_t k = 0; k < ns; k++) us[uint64_t(i) * ns + k] = double(T(ui[pm[k]]));
    });
    QSLC_CUDA(cudaMemcpyAsync(b->d_usorted, us.data(), us.size() * 8, cudaMemcpyHostToDevice, b->stream));
    QSLC_CUDA(cudaMemcpyAsync(b->d_perm, perm.data(), perm.size() * 4, cudaMemcpyHostToDevice, b->stream));
    QSLC_CUDA(cudaStreamSynchronize(b->stream));
    return QSLC_OK;
}

int upload_any(qslc_batch *b, const double *angles, const double *u)
{
    return b->dtype == QSLC_C128 ? upload_inputs<double>(b, angles, u) : upload_inputs<float>(b, angles, u);
}

int download(qslc_batch *b, double *probs, uint64_t *shots)
{
    QSLC_CUDA(cudaMemcpyAsync(probs, b->d_probs, b->nprobs * 8, cudaMemcpyDeviceToHost, b->stream));
    if (b->nshots)
        QSLC_CUDA(cudaMemcpyAsync(shots, b->d_shots, b->nshot_total * 8, cudaMemcpyDeviceToHost, b->stream));
    QSLC_CUDA(cudaStreamSynchronize(b->stream));
    QSLC_CUDA(cudaGetLastError());
    return QSLC_OK;
}

// The launch shapes the autotuner measures: threads per CTA, a tile of
// 64 or 128 KB, one or two CTAs per SM.
std::vector<BatchShape> candidates(const qslc_batch *b)
{
    const unsigned k128 = b->dtype == QSLC_C128 ? 13 : 14;
    std::vector<BatchShape> out;
    for (unsigned th : {512u, 1024u})
        for (const auto &tc : {std::pair<unsigned, unsigned>{k128 - 1, 2u}, {k128 - 1, 1u}, {k128, 1u}}) {
            BatchShape s;
            s.threads = th;
            s.tile_log2 = tc.first;
            s.ctas_per_sm = tc.second;
            if (shape_fits(b, s)) out.push_back(s);
        }
    return out;
}

}  // namespace

extern "C" int qslc_batch_create(int dtype, uint32_t ninst, const uint32_t *nqubits,
                                 const uint32_t *nlayers, uint32_t nshots, qslc_batch **out)
{
    QSLC_ENTRY("qslc_batch_create");
    if (!out || !nqubits || !nlayers || ninst == 0) return fail(QSLC_EINVAL, "bad batch arguments");
    *out = nullptr;
    if (dtype != QSLC_C128 && dtype != QSLC_C64) return fail(QSLC_EINVAL, "unknown dtype");
    auto *b = new qslc_batch();
    b->dtype = dtype;
    b->ninst = ninst;
    b->nshots = nshots;
    b->inst.resize(ninst);
    for (uint32_t i = 0; i < ninst; i++) {
        if (nqubits[i] < 2 || nqubits[i] > uint32_t(MAX_Q)) {
            delete b;
            return fail(QSLC_EINVAL, "batch instances take 2..26 qubits");
        }
        InstDesc &d = b->inst[i];
        d.n = nqubits[i];
        d.L = nlayers[i];
        d.coef = b->ncoef;
        d.probs = b->nprobs;
        d.shots = b->nshot_total;
        d.norms = b->nnorm_total;
        b->ncoef += uint64_t(d.L) * d.n * 4;
        b->nnorm_total += uint64_t(1) << d.n;
        b->nprobs += 2 * uint64_t(d.n);
        b->nshot_total += nshots;
        b->nmax = std::max(b->nmax, d.n);
    }
    // largest instances first, so the long ones start early
    b->order.resize(ninst);
    std::iota(b->order.begin(), b->order.end(), 0u);
    std::stable_sort(b->order.begin(), b->order.end(), [&](uint32_t x, uint32_t y) {
        return (uint64_t(b->inst[x].L) << b->inst[x].n) > (uint64_t(b->inst[y].L) << b->inst[y].n);
    });
    // the sums and CDF walks, one CTA per instance: the longest first
    b->size_order.resize(ninst);
    std::iota(b->size_order.begin(), b->size_order.end(), 0u);
    std::stable_sort(b->size_order.begin(), b->size_order.end(),
                     [&](uint32_t x, uint32_t y) { return b->inst[x].n > b->inst[y].n; });
    const size_t fb = dtype == QSLC_C128 ? 8 : 4;
    int rc = QSLC_OK;
    auto alloc = [&](void **p, size_t bytes) {
        if (rc) return;
        if (cudaMalloc(p, std::max<size_t>(bytes, 16)) != cudaSuccess) {
            cudaGetLastError();
            rc = fail(QSLC_EOOM, "out of device memory for the batch");
        }
    };
    alloc(&b->d_inst, ninst * sizeof(InstDesc));
    alloc(&b->d_order, ninst * 4);
    alloc(&b->d_counter, 16);
    alloc(&b->d_coef, b->ncoef * fb);
    alloc(&b->d_probs, b->nprobs * 8);
    alloc(&b->d_u, b->nshot_total * 8);
    alloc(&b->d_shots, b->nshot_total * 8);
    alloc(&b->d_usorted, b->nshot_total * 8);
    alloc(&b->d_perm, b->nshot_total * 4);
    alloc(&b->d_norms, b->nnorm_total * fb);
    alloc(&b->d_size_order, ninst * 4);
    alloc(&b->d_pick, size_t(sm_count()) * 8 * sizeof(unsigned));
    if (!rc && cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess)
        rc = fail(QSLC_ECUDA, "stream creation failed");
    // on the batch's own stream, which does not wait for the default one
    if (!rc && (cudaMemcpyAsync(b->d_inst, b->inst.data(), ninst * sizeof(InstDesc), cudaMemcpyHostToDevice,
                                b->stream) != cudaSuccess ||
                cudaMemcpyAsync(b->d_size_order, b->size_order.data(), ninst * 4, cudaMemcpyHostToDevice,
                                b->stream) != cudaSuccess))
        rc = fail(QSLC_ECUDA, "upload failed");
    if (!rc && (cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking) != cudaSuccess ||
                cudaEventCreateWithFlags(&b->forked, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&b->joined, cudaEventDisableTiming) != cudaSuccess))
        rc = fail(QSLC_ECUDA, "stream creation failed");
    if (!rc) {
        const auto c = candidates(b);
        if (c.empty()) rc = fail(QSLC_EINVAL, "no launch shape fits the largest instance");
        else {
            // the 128 KB tile: for complex64 with 512 threads of 128
            // registers (4096 instances 171 ms, with 1024 of 64 183), for
            // complex128 with 1024
            const BatchShape *s = &c.back();
            for (const BatchShape &k : c)
                if (dtype == QSLC_C64 && k.threads == 512 && k.tile_log2 == c.back().tile_log2) s = &k;
            rc = capture_any(b, *s);
        }
    }
    if (rc) {
        batch_free(b);
        return rc;
    }
    *out = b;
    return QSLC_OK;
}

extern "C" int qslc_batch_run(qslc_batch *b, const double *angles, const double *uniforms,
                              double *probs, uint64_t *shots)
{
    QSLC_ENTRY("qslc_batch_run");
    if (!b || !angles || !probs || (!uniforms && b->nshots) || (!shots && b->nshots))
        return fail(QSLC_EINVAL, "null pointer");
    int rc = upload_any(b, angles, uniforms);
    if (rc) return rc;
    QSLC_CUDA(cudaGraphLaunch(b->exec, b->stream));
    rc = download(b, probs, shots);
    if (!rc) b->runs++;
    return rc;
}

extern "C" int qslc_batch_autotune(qslc_batch *b, const double *angles, const double *uniforms,
                                   double *best_ms)
{
    QSLC_ENTRY("qslc_batch_autotune");
    if (!b || !angles || (!uniforms && b->nshots)) return fail(QSLC_EINVAL, "null pointer");
    int rc = upload_any(b, angles, uniforms);
    if (rc) return rc;
    cudaEvent_t e0, e1;
    QSLC_CUDA(cudaEventCreate(&e0));
    QSLC_CUDA(cudaEventCreate(&e1));
    BatchShape best = b->shape;
    float best_t = -1.f;
    for (const BatchShape &s : candidates(b)) {
        rc = capture_any(b, s);
        if (rc) break;
        QSLC_CUDA(cudaGraphLaunch(b->exec, b->stream));        // warm-up
        QSLC_CUDA(cudaEventRecord(e0, b->stream));
        QSLC_CUDA(cudaGraphLaunch(b->exec, b->stream));
        QSLC_CUDA(cudaEventRecord(e1, b->stream));
        QSLC_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        QSLC_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (best_t < 0.f || ms < best_t) {
            best_t = ms;
            best = s;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!rc) rc = capture_any(b, best);
    if (!rc && best_ms) *best_ms = double(best_t);
    return rc;
}

extern "C" int qslc_batch_set_shape(qslc_batch *b, unsigned threads, unsigned tile_log2,
                                    unsigned ctas_per_sm)
{
    QSLC_ENTRY("qslc_batch_set_shape");
    if (!b) return fail(QSLC_EINVAL, "null batch");
    BatchShape s;
    s.threads = threads;
    s.tile_log2 = tile_log2;
    s.ctas_per_sm = ctas_per_sm;
    for (const BatchShape &c : candidates(b))
        if (c.threads == s.threads && c.tile_log2 == s.tile_log2 && c.ctas_per_sm == s.ctas_per_sm)
            return capture_any(b, s);
    return fail(QSLC_EINVAL, "not one of the launch shapes this batch can take");
}

extern "C" int qslc_batch_shape(const qslc_batch *b, unsigned *threads, unsigned *tile_log2,
                                unsigned *ctas_per_sm, unsigned *grid)
{
    QSLC_ENTRY("qslc_batch_shape");
    if (!b) return fail(QSLC_EINVAL, "null batch");
    if (threads) *threads = b->shape.threads;
    if (tile_log2) *tile_log2 = b->shape.tile_log2;
    if (ctas_per_sm) *ctas_per_sm = b->shape.ctas_per_sm;
    if (grid) *grid = b->grid;
    return QSLC_OK;
}

extern "C" int qslc_batch_destroy(qslc_batch *b)
{
    batch_free(b);
    return QSLC_OK;
}
