// run.cu -- runs of gates in one sweep of the state.
//
// Gates on a plain state are queued, and a run of consecutive gates whose
// qubits fit one tile is applied by one kernel: a CTA copies a tile of 2^B
// amplitudes -- all combinations of the B tile qubits, the other qubits
// fixed -- into shared memory, applies the gates one after the other with a
// barrier between them, and copies the tile back.  Each gate acts on every
// tile as its own sweep would act on the state (a tile holds both members of
// every pair), with the same operations in the same order on each amplitude,
// so the bits are those of the single sweeps.  What changes is the traffic:
// the state is read and written once for the run instead of once per gate,
// and one launch takes the place of many.
//
// The tile qubits always include the lowest ones (L of them), so a tile is
// made of contiguous pieces of 2^L amplitudes.  Only the qubits along which a
// gate mixes amplitudes need to be in the tile: controls and the targets of
// diagonal gates are tested on the indices.
//
// complex64 sweeps are bound by HBM one gate at a time, and runs by
// instructions: four layers of a 25-qubit circuit take 2.3 ms, 5.6 ms with a
// sweep for two gates.  complex128 runs are bound by the FP64 and ALU pipes as the
// single sweeps are, and gain where launches or moves count: 8 layers of 10
// qubits, 120 calls, 418 -> 165 us.
#include "bounds.cuh"
#include "gatemath.cuh"

#include <algorithm>
#include <atomic>
#include <vector>

namespace qslc {
namespace {

constexpr int RUN_MAX_BITS = 12;       // 64 KB of complex128, 32 KB of complex64
constexpr int RUN_LOADS = 8;           // amplitudes a thread loads before it stores them to shared memory
constexpr int RUN_CTAS = 4;            // CTAs of 256 threads per SM: 64 registers a thread
constexpr int RUN_MAX_GATES = 48;      // lowered gates of one run

// A lowered gate.  Pair gates (swap of the pair, Y, H, RX, RY) act on the
// pairs along register bit `p` whose number is in `set`; diagonal ones on the
// amplitudes whose number is in `set`.  Both only where the tile-local index
// has all bits of `lmask` and the tile's own index all of `gmask`: a control
// need not be in registers, nor even in the tile, and neither need the
// target of a diagonal gate.  ROTATE is phase's update (x c - y s, y c + x s)
// with s negated for the amplitudes in `neg`, and for all of them where the
// bit of `lflip` or `gflip` is clear (rotateZ on the |0> members).
enum RunOp : uint8_t { RUN_SWAP, RUN_Y, RUN_H, RUN_RX, RUN_RY, RUN_NEG, RUN_ROTATE };

struct alignas(16) RunGate {
    uint8_t op, p;
    uint16_t set, neg;
    uint16_t lmask, lflip;
    uint16_t outside;        // 1: gmask or gflip is not zero
    uint32_t pad;
    uint64_t gmask, gflip;
};

// Consecutive gates that share a choice of register bits.
struct RunStep {
    uint8_t bit[4];      // tile-local bits, ascending
    uint8_t first, count;
};

template <class T> struct RunCoef;
template <> struct RunCoef<float> {
    float c, s;
};
template <> struct RunCoef<double> {
    double c, s;
    emu::MulK mc, ms;
    emu::LeanK lc, ls;
};
static_assert(offsetof(RunCoef<double>, ms) == offsetof(SlowCoef, ms), "SlowCoef heads RunCoef<double>");

// Register bits of a thread: 4 amplitudes of 16 bytes or 16 of 8, and on small
// states 2 of 16 bytes or 4 of 8 (reg_bits).
template <class T> constexpr int REG_BITS = sizeof(T) == 8 ? 2 : 4;
template <class T> constexpr int SMALL_REG_BITS = sizeof(T) == 8 ? 1 : 2;

template <class T, int NG>
struct RunArgs {
    uint64_t ntiles;
    uint64_t chunk[32];                // offset of a tile's amplitudes i * threads
    uint8_t pos[RUN_MAX_BITS + 4];     // the state's bit of each tile bit, ascending
    uint8_t bits, low, nsteps;
    Coef<T> h;                         // Hadamard's constants
    float hinv;                        // RN(1 / sqrt(2)) for complex64
    RunStep step[NG];
    RunGate gate[NG];
    RunCoef<T> coef[NG];
};

// Where local amplitude l lies in shared memory: its low bits are mixed
// with the next ones, so that the lanes of one access, whose indices skip a
// register bit, fall in different banks for most choices of those bits.
template <class T>
__device__ __forceinline__ uint32_t slot_of(uint32_t l)
{
    if constexpr (sizeof(T) == 8) return l ^ ((0x2570u >> (4 * ((l >> 3) & 3u))) & 7u);
    else return l ^ ((l >> 4) & 15u);
}

// ---- complex128: 2 or 4 amplitudes -------------------------------------------

template <int OP, int A>
__device__ __forceinline__ void run_pairs(double2 (&v)[A], unsigned set, const Coef<double> &k, const SlowCoef *q,
                                          const emu::DivConst *kd)
{
    auto pair = [&](double2 &a0, double2 &a1) {
        if constexpr (OP == P_SWAP || OP == P_Y) pair_update<double, OP>(a0, a1, k);
        else pair_either<OP>(a0, a1, k, q, kd);
    };
    if constexpr (A == 2) {
        pair(v[0], v[1]);
    } else if (set == 3) {
        pair(v[0], v[1]);
        pair(v[2], v[3]);
    } else if (set == 1) {
        pair(v[0], v[1]);
    } else {
        pair(v[2], v[3]);
    }
}

__device__ __forceinline__ void run_rotate(double2 &a, uint32_t flip, const Coef<double> &k, const SlowCoef *q)
{
    phase_flip(a, flip, k, q);
}

template <int A, int NG>
__device__ __forceinline__ void run_gate(double2 (&v)[A], const RunGate &g, const RunCoef<double> &r, bool flip_all,
                                         const RunArgs<double, NG> &a)
{
    Coef<double> k{};
    k.c = g.op == RUN_H ? a.h.c : r.c;
    k.s = r.s;
    k.lc = r.lc;
    k.ls = r.ls;
    k.ld = a.h.ld;
    const SlowCoef *q = reinterpret_cast<const SlowCoef *>(&r);
    if (g.op >= RUN_NEG) {
#pragma unroll
        for (int i = 0; i < A; i++) {
            if (!((g.set >> i) & 1)) continue;
            if (g.op == RUN_NEG) diag_update<double, D_NEG>(v[i], k);
            else run_rotate(v[i], (((g.neg >> i) & 1) != 0) != flip_all ? 0x80000000u : 0u, k, q);
        }
        return;
    }
    auto turn = [&] {
        if constexpr (A == 4)
            if (g.p) {
                const double2 m = v[1];
                v[1] = v[2];
                v[2] = m;
            }
    };
    turn();
    switch (g.op) {
    case RUN_SWAP: run_pairs<P_SWAP>(v, g.set, k, q, &a.h.kd); break;
    case RUN_Y: run_pairs<P_Y>(v, g.set, k, q, &a.h.kd); break;
    case RUN_H: run_pairs<P_H>(v, g.set, k, q, &a.h.kd); break;
    case RUN_RX: run_pairs<P_RX>(v, g.set, k, q, &a.h.kd); break;
    default: run_pairs<P_RY>(v, g.set, k, q, &a.h.kd); break;
    }
    turn();
}

// ---- complex64: 4 or 16 amplitudes -------------------------------------------

template <int OP, int P, bool ALL, int A>
__device__ __forceinline__ void run_pairs_on(float2 (&v)[A], unsigned set, const Coef<float> &k, float hinv)
{
#pragma unroll
    for (int i = 0; i < A / 2; i++) {
        const int i0 = ((i >> P) << (P + 1)) | (i & ((1 << P) - 1)), i1 = i0 | (1 << P);
        if (!ALL && !((set >> i) & 1)) continue;
        if constexpr (OP == P_H) {
            const float2 a = v[i0], b = v[i1];
            const float s0 = __fadd_rn(a.x, b.x), s1 = __fadd_rn(a.y, b.y);
            const float d0 = __fsub_rn(a.x, b.x), d1 = __fsub_rn(a.y, b.y);
            v[i0] = make_float2(emu::div_step(s0, k.c, hinv), emu::div_step(s1, k.c, hinv));
            v[i1] = make_float2(emu::div_step(d0, k.c, hinv), emu::div_step(d1, k.c, hinv));
            const float lo = fminf(fminf(fabsf(s0), fabsf(s1)), fminf(fabsf(d0), fabsf(d1)));
            const float hi = fmaxf(fmaxf(fabsf(s0), fabsf(s1)), fmaxf(fabsf(d0), fabsf(d1)));
            if (!(lo >= 0x1p-100f && hi <= 0x1.fffffep127f)) {
                if (!emu::div_step_takes(s0)) v[i0].x = __fdiv_rn(s0, k.c);
                if (!emu::div_step_takes(s1)) v[i0].y = __fdiv_rn(s1, k.c);
                if (!emu::div_step_takes(d0)) v[i1].x = __fdiv_rn(d0, k.c);
                if (!emu::div_step_takes(d1)) v[i1].y = __fdiv_rn(d1, k.c);
            }
        } else {
            pair_update<float, OP>(v[i0], v[i1], k);
        }
    }
}

template <int OP, bool ALL, int A>
__device__ __forceinline__ void run_pairs_at(float2 (&v)[A], int p, unsigned set, const Coef<float> &k, float hinv)
{
    if constexpr (A == 4) {
        if (p == 0) run_pairs_on<OP, 0, ALL>(v, set, k, hinv);
        else run_pairs_on<OP, 1, ALL>(v, set, k, hinv);
    } else {
        switch (p) {
        case 0: run_pairs_on<OP, 0, ALL>(v, set, k, hinv); break;
        case 1: run_pairs_on<OP, 1, ALL>(v, set, k, hinv); break;
        case 2: run_pairs_on<OP, 2, ALL>(v, set, k, hinv); break;
        default: run_pairs_on<OP, 3, ALL>(v, set, k, hinv); break;
        }
    }
}

template <bool ALL, int A>
__device__ __forceinline__ void run_rotate_on(float2 (&v)[A], unsigned set, unsigned neg, bool flip_all,
                                             const Coef<float> &k)
{
    const float sp = flip_all ? -k.s : k.s;
#pragma unroll
    for (int i = 0; i < A; i++) {
        if (!ALL && !((set >> i) & 1)) continue;
        const float s = ((neg >> i) & 1) ? -sp : sp;
        const float x = v[i].x, y = v[i].y;
        v[i].x = __fsub_rn(__fmul_rn(x, k.c), __fmul_rn(y, s));
        v[i].y = __fadd_rn(__fmul_rn(y, k.c), __fmul_rn(x, s));
    }
}

template <int A, int NG>
__device__ __forceinline__ void run_gate(float2 (&v)[A], const RunGate &g, const RunCoef<float> &r, bool flip_all,
                                         const RunArgs<float, NG> &a)
{
    Coef<float> k{};
    k.c = g.op == RUN_H ? a.h.c : r.c;
    k.s = r.s;
    const bool all = g.set == (1u << (A / 2)) - 1u;
    switch (g.op) {
    case RUN_SWAP: run_pairs_at<P_SWAP, false>(v, g.p, g.set, k, 0.f); break;
    case RUN_Y: run_pairs_at<P_Y, false>(v, g.p, g.set, k, 0.f); break;
    case RUN_H:
        if (all) run_pairs_at<P_H, true>(v, g.p, g.set, k, a.hinv);
        else run_pairs_at<P_H, false>(v, g.p, g.set, k, a.hinv);
        break;
    case RUN_RX:
        if (all) run_pairs_at<P_RX, true>(v, g.p, g.set, k, 0.f);
        else run_pairs_at<P_RX, false>(v, g.p, g.set, k, 0.f);
        break;
    case RUN_RY:
        if (all) run_pairs_at<P_RY, true>(v, g.p, g.set, k, 0.f);
        else run_pairs_at<P_RY, false>(v, g.p, g.set, k, 0.f);
        break;
    case RUN_NEG:
#pragma unroll
        for (int i = 0; i < A; i++)
            if ((g.set >> i) & 1) diag_update<float, D_NEG>(v[i], k);
        break;
    default:
        if (g.set == (1u << A) - 1u) run_rotate_on<true>(v, g.set, g.neg, flip_all, k);
        else run_rotate_on<false>(v, g.set, g.neg, flip_all, k);
        break;
    }
}

template <class T, class IX, int NG, int R>
__global__ void __launch_bounds__(256, RUN_CTAS)
    k_run(cplx<T> *__restrict__ st, const __grid_constant__ RunArgs<T, NG> a)
{
    extern __shared__ __align__(128) unsigned char run_smem[];
    constexpr int A = 1 << R;
    constexpr uint32_t AB = sizeof(cplx<T>);
    auto at = [&](uint32_t byte) -> cplx<T> & { return *reinterpret_cast<cplx<T> *>(run_smem + byte); };
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    const uint32_t size = 1u << a.bits;
    const int rounds = int(size / nt);
    IX mine = 0;                                   // offset of amplitude tid of a tile
    for (int i = 0; (1u << i) < nt; i++) mine |= IX((tid >> i) & 1u) << a.pos[i];
    const uint32_t home = slot_of<T>(tid) * AB;    // slot_of is linear: tid + i nt lies at home ^ slot_of(i nt)
    for (uint64_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
        IX tile = IX(t) << a.low;
        for (int i = a.low; i < a.bits; i++) tile = ins0<IX>(tile, a.pos[i]);
        cplx<T> *const mem = st + (tile | mine);
        for (int i0 = 0; i0 < rounds; i0 += RUN_LOADS) {
            cplx<T> v[RUN_LOADS];
#pragma unroll
            for (int u = 0; u < RUN_LOADS; u++)
                if (i0 + u < rounds && QSLC_IN_STATE((tile | mine) + a.chunk[i0 + u], a.ntiles << a.bits))
                    v[u] = mem[a.chunk[i0 + u]];
#pragma unroll
            for (int u = 0; u < RUN_LOADS; u++)
                if (i0 + u < rounds && QSLC_IN_STATE_QUIET((tile | mine) + a.chunk[i0 + u], a.ntiles << a.bits))
                    at(home ^ (slot_of<T>((i0 + u) * nt) * AB)) = v[u];
        }
        __syncthreads();
        for (int s = 0; s < a.nsteps; s++) {
            const RunStep sp = a.step[s];
            uint32_t off[R];
#pragma unroll
            for (int i = 0; i < R; i++) off[i] = slot_of<T>(1u << sp.bit[i]) * AB;
            for (uint32_t q = tid; q < size >> R; q += nt) {
                uint32_t l = q;
#pragma unroll
                for (int i = 0; i < R; i++) l = ins0<uint32_t>(l, sp.bit[i]);
                const uint32_t x = slot_of<T>(l) * AB;
                auto addr = [&](int i) {
                    uint32_t o = 0;
#pragma unroll
                    for (int b = 0; b < R; b++)
                        if (i & (1 << b)) o ^= off[b];
                    return x ^ o;
                };
                cplx<T> v[A];
#pragma unroll
                for (int i = 0; i < A; i++) v[i] = at(addr(i));
#pragma unroll 1
                for (int g = sp.first; g < sp.first + sp.count; g++) {
                    const RunGate &rg = a.gate[g];
                    if ((l & rg.lmask) != rg.lmask) continue;
                    bool flip_all = rg.lflip && !(l & rg.lflip);
                    if (rg.outside) {
                        if ((uint64_t(tile) & rg.gmask) != rg.gmask) continue;
                        flip_all = flip_all || (rg.gflip && !(uint64_t(tile) & rg.gflip));
                    }
                    run_gate(v, rg, a.coef[g], flip_all, a);
                }
#pragma unroll
                for (int i = 0; i < A; i++) at(addr(i)) = v[i];
            }
            __syncthreads();
        }
        for (int i0 = 0; i0 < rounds; i0 += RUN_LOADS) {
#pragma unroll
            for (int u = 0; u < RUN_LOADS; u++)
                if (i0 + u < rounds && QSLC_IN_STATE_QUIET((tile | mine) + a.chunk[i0 + u], a.ntiles << a.bits))
                    mem[a.chunk[i0 + u]] = at(home ^ (slot_of<T>((i0 + u) * nt) * AB));
        }
    }
}

// The tile of a state: log2 of its amplitudes, contiguous low bits, threads.
struct Shape {
    unsigned bits, low, threads;
};

// The register bits of a thread.  A small state leaves most of the chip idle,
// and a gate takes the time that one warp needs for its amplitudes, about 8
// clocks an instruction: fewer amplitudes a thread, in more warps, are quicker
// although the targets of a run then take more steps.  Circuits of 8 layers, us,
// usual and small: complex128 of 6 qubits 140 and 106, of 10 195 and 162, of 14
// 275 and 214, of 17 372 and 308, of 18 462 and 428, of 19 626 and 716; complex64
// of 6 qubits 96 and 87, of 12 172 and 163, of 14 (usual) 197.
template <class T> constexpr unsigned FEW_REGS = sizeof(T) == 8 ? 18 : 13;
template <class T> int reg_bits(const qslc_state *s)
{
    return s->n <= FEW_REGS<T> ? SMALL_REG_BITS<T> : REG_BITS<T>;
}

// complex128 states of this many qubits take runs of everything (runs_any).
constexpr unsigned SMALL_STATE = 19;

// Small states take small tiles: many CTAs share the arithmetic, which a run
// of few gates does not fill otherwise.  Circuits of 8 layers on one GB300,
// us, tiles of 2^7 / 2^8 / 2^9 / 2^10 amplitudes: complex128 of 10 qubits 167 /
// 162 / 162 / 235, of 14 231 / 218 / 215 / 308, of 17 325 / 308 / 297 / 387, of 19
// with 2^8 627, with 2^11 748; complex64 of 10 qubits 145 / 140 / 135 / 129, of 14
// 215 / 201 / 200 / 192, of 25 (4 layers) 3044 with 2^10, 2871 with 2^11 and 2655
// with 2^12.  Two contiguous low qubits were never slower than three or four: the
// others are left to the run.
Shape shape_of(const qslc_state *s)
{
    const bool dbl = s->dtype == QSLC_C128;
    const unsigned b = std::min(dbl ? (s->n > SMALL_STATE ? 11u : 8u) : (s->n >= 20 ? 12u : 10u), s->n);
    const unsigned r = unsigned(dbl ? reg_bits<double>(s) : reg_bits<float>(s));
    const unsigned t = b >= r + 8 ? 256 : b > r + 5 ? 1u << (b - r) : 32;
    return Shape{b, std::min(b, 2u), std::min(t, 1u << b)};
}

// A gate in the kernel's terms: an update on target t where control c is set
// (NO_QUBIT: no control).
constexpr unsigned NO_QUBIT = 64;

template <class T>
struct Lowered {
    RunOp op;
    unsigned t, c;
    bool both;            // rotateZ: the |0> members too, with s negated
    RunCoef<T> coef;
};

template <class T>
RunCoef<T> pack(const Coef<T> &k)
{
    RunCoef<T> r{};
    r.c = k.c;
    r.s = k.s;
    if constexpr (sizeof(T) == 8) {
        r.mc = k.mc;
        r.ms = k.ms;
        r.lc = k.lc;
        r.ls = k.ls;
    }
    return r;
}

// The exchanges (swap, npRotateX, ...) act on the members (q1 set, q2 clear)
// and (q1 clear, q2 set): controlNot(q2, q1) brings the second to (both set),
// the update then is one on q2 controlled by q1, and a second controlNot
// brings it back.  Moves are exact, so the bits are the same.
template <class T>
void lower(const GateOp &g, std::vector<Lowered<T>> &out)
{
    const Coef<T> none{};
    auto put = [&](RunOp op, unsigned t, unsigned c, const Coef<T> &k, bool both = false) {
        out.push_back(Lowered<T>{op, t, c, both, pack<T>(k)});
    };
    auto one = [&](RunOp op, const Coef<T> &k, bool both = false) { put(op, g.q1, NO_QUBIT, k, both); };
    auto ctrl = [&](RunOp op, const Coef<T> &k, bool both = false) { put(op, g.q2, g.q1, k, both); };
    auto xchg = [&](RunOp op, const Coef<T> &k) {
        put(RUN_SWAP, g.q1, g.q2, none);
        put(op, g.q2, g.q1, k);
        put(RUN_SWAP, g.q1, g.q2, none);
    };
    switch (g.code) {
    case QSLC_PAULI_X: one(RUN_SWAP, none); break;
    case QSLC_PAULI_Y: one(RUN_Y, none); break;
    case QSLC_PAULI_Z: one(RUN_NEG, none); break;
    case QSLC_HADAMARD: one(RUN_H, none); break;
    case QSLC_PHASE: one(RUN_ROTATE, full_angle<T>(g.angle)); break;
    case QSLC_ROTATE_X: one(RUN_RX, half_angle<T>(g.angle)); break;
    case QSLC_ROTATE_Y: one(RUN_RY, half_angle<T>(g.angle)); break;
    case QSLC_ROTATE_Z: one(RUN_ROTATE, half_angle<T>(g.angle), true); break;
    case QSLC_CONTROL_NOT: ctrl(RUN_SWAP, none); break;
    case QSLC_CONTROL_Y: ctrl(RUN_Y, none); break;
    case QSLC_CONTROL_Z: ctrl(RUN_NEG, none); break;
    case QSLC_CONTROL_ROTATE_X: ctrl(RUN_RX, half_angle<T>(g.angle)); break;
    case QSLC_CONTROL_ROTATE_Y: ctrl(RUN_RY, half_angle<T>(g.angle)); break;
    case QSLC_CONTROL_ROTATE_Z: ctrl(RUN_ROTATE, half_angle<T>(g.angle), true); break;
    case QSLC_CONTROL_PHASE: ctrl(RUN_ROTATE, full_angle<T>(g.angle)); break;
    case QSLC_CONTROL_HADAMARD: ctrl(RUN_H, none); break;
    case QSLC_SWAP: xchg(RUN_SWAP, none); break;
    case QSLC_FSWAP:
        xchg(RUN_SWAP, none);
        ctrl(RUN_NEG, none);
        break;
    case QSLC_NP_ROTATE_X: xchg(RUN_RX, half_angle<T>(g.angle)); break;
    case QSLC_NP_ROTATE_Y: xchg(RUN_RY, half_angle<T>(g.angle)); break;
    default: xchg(RUN_H, none); break;     // QSLC_NP_HADAMARD
    }
}

bool is_diagonal(RunOp op) { return op >= RUN_NEG; }

// The kernel's view of gate o in a step with register bits `reg` (state
// qubits; reg[i] is register bit i) of a tile whose qubits' local numbers are
// `local` (0xFF: not in the tile).
template <class T, int R>
RunGate encode(const Lowered<T> &o, const unsigned *reg, const uint8_t *local)
{
    constexpr int A = 1 << R;
    RunGate g{};
    g.op = o.op;
    auto reg_bit = [&](unsigned q) {
        for (int i = 0; i < R; i++)
            if (reg[i] == q) return i;
        return -1;
    };
    unsigned amps = (1u << A) - 1;            // the register amplitudes the gate touches
    auto require = [&](unsigned q) {          // only where qubit q is set
        const int r = reg_bit(q);
        if (r >= 0) {
            for (int i = 0; i < A; i++)
                if (!((i >> r) & 1)) amps &= ~(1u << i);
        } else if (local[q] != 0xFF) g.lmask |= uint16_t(1u << local[q]);
        else g.gmask |= uint64_t(1) << q;
    };
    if (o.c != NO_QUBIT) require(o.c);
    if (is_diagonal(o.op)) {
        if (!o.both) require(o.t);
        else {
            const int r = reg_bit(o.t);
            if (r >= 0) {
                for (int i = 0; i < A; i++)
                    if (!((i >> r) & 1)) g.neg |= uint16_t(1u << i);
            } else if (local[o.t] != 0xFF) g.lflip = uint16_t(1u << local[o.t]);
            else g.gflip = uint64_t(1) << o.t;
        }
        g.set = uint16_t(amps);
    } else {
        const int p = reg_bit(o.t);
        g.p = uint8_t(p);
        for (int i = 0; i < A / 2; i++) {
            const int i0 = ((i >> p) << (p + 1)) | (i & ((1 << p) - 1));
            if ((amps >> i0) & 1) g.set |= uint16_t(1u << i);
        }
    }
    g.outside = (g.gmask | g.gflip) != 0;
    return g;
}

template <class T, int NG, int R>
int launch_run_t(qslc_state *s, const std::vector<Lowered<T>> &ops, uint64_t mask)
{
    const Shape sh = shape_of(s);
    static const Coef<T> hcoef = sqrt2_coef<T>();
    RunArgs<T, NG> a;
    a.bits = uint8_t(sh.bits);
    a.low = uint8_t(sh.low);
    // tile qubits: the run's, the lowest ones, and the lowest unused ones to fill up
    mask |= (uint64_t(1) << sh.low) - 1;
    for (unsigned q = 0; unsigned(__builtin_popcountll(mask)) < sh.bits; q++) mask |= uint64_t(1) << q;
    uint8_t local[65];
    std::fill(local, local + 65, uint8_t(0xFF));
    unsigned at = 0;
    for (unsigned q = 0; q < s->n; q++)
        if ((mask >> q) & 1) {
            local[q] = uint8_t(at);
            a.pos[at++] = uint8_t(q);
        }
    const unsigned lt = unsigned(__builtin_ctz(sh.threads));
    for (unsigned i = 0; i < (1u << (sh.bits - lt)); i++) {
        uint64_t o = 0;
        for (unsigned k = 0; k < sh.bits - lt; k++)
            if ((i >> k) & 1) o |= uint64_t(1) << a.pos[lt + k];
        a.chunk[i] = o;
    }
    a.h = hcoef;
    a.hinv = 1.0f / float(hcoef.c);
    a.nsteps = 0;
    for (size_t i = 0; i < ops.size();) {
        // as many gates as have their targets in R register bits
        unsigned reg[R];
        int nreg = 0;
        size_t j = i;
        for (; j < ops.size(); j++) {
            if (is_diagonal(ops[j].op)) continue;
            if (std::find(reg, reg + nreg, ops[j].t) != reg + nreg) continue;
            if (nreg == R) break;
            reg[nreg++] = ops[j].t;
        }
        // the other register bits: first the qubits of controls and diagonal
        // gates that would tell the lanes of a warp apart, then the tile's
        // highest unused ones
        for (unsigned k = 0; k < 5 && k < sh.bits && nreg < R; k++) {
            const unsigned q = a.pos[k];
            if (std::find(reg, reg + nreg, q) != reg + nreg) continue;
            for (size_t g = i; g < j; g++)
                if (ops[g].c == q || (is_diagonal(ops[g].op) && ops[g].t == q)) {
                    reg[nreg++] = q;
                    break;
                }
        }
        for (int k = int(sh.bits) - 1; nreg < R; k--)
            if (std::find(reg, reg + nreg, unsigned(a.pos[k])) == reg + nreg) reg[nreg++] = a.pos[k];
        std::sort(reg, reg + R);
        RunStep &sp = a.step[a.nsteps++];
        sp.first = uint8_t(i);
        sp.count = uint8_t(j - i);
        for (int k = 0; k < R; k++) sp.bit[k] = local[reg[k]];
        for (; i < j; i++) {
            a.gate[i] = encode<T, R>(ops[i], reg, local);
            a.coef[i] = ops[i].coef;
        }
    }
    a.ntiles = uint64_t(1) << (s->n - sh.bits);
    const size_t smem = sizeof(cplx<T>) << sh.bits;
    auto go = [&](auto ix) -> int {
        using IX = decltype(ix);
        auto *kern = k_run<T, IX, NG, R>;
        static std::atomic<int> per_sm[RUN_MAX_BITS + 1] = {};
        if (!per_sm[sh.bits]) {
            QSLC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(sizeof(cplx<T>) << RUN_MAX_BITS)));
            int b = 0;
            QSLC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, int(sh.threads), smem));
            if (b < 1) return fail(QSLC_ECUDA, "a run's tile does not fit on an SM");
            per_sm[sh.bits] = b;
        }
        const uint64_t grid = std::min<uint64_t>(a.ntiles, uint64_t(sm_count()) * unsigned(per_sm[sh.bits].load()));
        kern<<<unsigned(grid), sh.threads, smem, s->stream>>>(static_cast<cplx<T> *>(s->amps), a);
        return QSLC_OK;
    };
    int rc;
    if constexpr (R == SMALL_REG_BITS<T>) rc = go(uint32_t(0));
    else rc = s->n <= 31 ? go(uint32_t(0)) : go(uint64_t(0));
    if (rc) return rc;
    s->launches++;
    QSLC_CUDA(cudaGetLastError());
    return QSLC_OK;
}

template <class T>
int launch_run(qslc_state *s, const std::vector<GateOp> &gates, uint64_t mask)
{
    std::vector<Lowered<T>> ops;
    for (const GateOp &g : gates) lower<T>(g, ops);
    if (reg_bits<T>(s) == SMALL_REG_BITS<T>)
        return ops.size() <= 16 ? launch_run_t<T, 16, SMALL_REG_BITS<T>>(s, ops, mask)
                                : launch_run_t<T, RUN_MAX_GATES, SMALL_REG_BITS<T>>(s, ops, mask);
    return ops.size() <= 16 ? launch_run_t<T, 16, REG_BITS<T>>(s, ops, mask)
                            : launch_run_t<T, RUN_MAX_GATES, REG_BITS<T>>(s, ops, mask);
}

// The qubits a gate needs in the tile: those along which it mixes amplitudes.
uint64_t qubits_of(const GateOp &g)
{
    const uint64_t b1 = uint64_t(1) << g.q1, b2 = uint64_t(1) << g.q2;
    switch (g.code) {
    case QSLC_PAULI_Z: case QSLC_PHASE: case QSLC_ROTATE_Z:
    case QSLC_CONTROL_Z: case QSLC_CONTROL_PHASE: case QSLC_CONTROL_ROTATE_Z:
        return 0;
    case QSLC_SWAP: case QSLC_FSWAP: case QSLC_NP_ROTATE_X: case QSLC_NP_ROTATE_Y: case QSLC_NP_HADAMARD:
        return b1 | b2;
    default:
        return b2;       // q2 == q1 for a one-qubit gate
    }
}

size_t lowered_of(int code)
{
    return code == QSLC_FSWAP ? 4 : code == QSLC_SWAP || code >= QSLC_NP_ROTATE_X ? 3 : 1;
}

// Two-qubit gates that only move amplitudes, change signs or rotate a
// quarter of the state: on a large complex128 state the rest is bound by
// arithmetic, which register sweeps do faster.
bool is_move(int code)
{
    switch (code) {
    case QSLC_CONTROL_NOT: case QSLC_CONTROL_Y: case QSLC_CONTROL_Z: case QSLC_CONTROL_PHASE:
    case QSLC_SWAP: case QSLC_FSWAP:
        return true;
    default:
        return false;
    }
}

// Whether runs take any gate: complex64 states, and complex128 ones small
// enough for launches to count more than arithmetic.  On larger ones the
// arithmetic binds, and a rotation takes 1.71 clocks per amplitude and SM in a
// run (coefficients read per gate, a barrier per two gates) against 1.29 in
// k_group2.  Circuits of 8 layers, us, pairs with runs of moves beside them
// against runs of everything: of one-qubit gates and all two-qubit gates, 18 qubits
// 796 and 504, 19 qubits 1090 and 835; of one-qubit gates and controlNots, 18 qubits
// 682 and 428, 19 qubits 919 and 627, 20 qubits 1209 and 1248.
bool runs_any(const qslc_state *s) { return s->dtype == QSLC_C64 || s->n <= SMALL_STATE; }

// Whether one run is quicker than the gates' own sweeps, by the share of the
// state that each moves (in quarters of a read and write of all of it) and,
// in a run, a gate's own time in the same unit: at 26 qubits a controlNot adds
// 76 us to a complex128 run and 24 us to a complex64 one, whose sweeps of the
// whole state take 320 and 160 us.  States below 18 qubits are bound by launches:
// any two gates but the pairs that k_group2 takes.
bool run_pays(const qslc_state *s, const std::vector<GateOp> &gates)
{
    if (s->n < 18) return !(gates.size() == 2 && !is_two_qubit(gates[0].code) && !is_two_qubit(gates[1].code));
    double alone = 0, run = 4;
    bool one = false;
    for (const GateOp &g : gates) {
        switch (g.code) {
        case QSLC_PHASE: case QSLC_PAULI_Z: alone += 2; break;
        case QSLC_CONTROL_Z: case QSLC_CONTROL_PHASE: alone += 1.2; break;
        case QSLC_FSWAP: alone += 3; break;
        default: alone += is_two_qubit(g.code) ? 2 : one ? 0 : 4; break;
        }
        one = !is_two_qubit(g.code) && !one;      // the next one-qubit gate would join this one
        if (s->dtype == QSLC_C128) run += g.code == QSLC_CONTROL_PHASE ? 1.3 : lowered_of(g.code);
        else run += 0.6 * double(lowered_of(g.code));
    }
    return run < alone;
}

// The gates one by one, one-qubit gates on different qubits two to a sweep.
int launch_each(qslc_state *s, const std::vector<GateOp> &gates)
{
    for (size_t i = 0; i < gates.size(); i++) {
        const GateOp &g = gates[i];
        int rc;
        if (is_two_qubit(g.code)) rc = launch_gate2(s, g.code, g.q1, g.q2, g.angle);
        else if (i + 1 < gates.size() && !is_two_qubit(gates[i + 1].code) && gates[i + 1].q1 != g.q1) {
            rc = launch_group2(s, g, gates[i + 1]);
            i++;
        } else
            rc = launch_gate1(s, g.code, g.q1, g.angle);
        if (rc) return rc;
    }
    return QSLC_OK;
}

}  // namespace

int run_release(qslc_state *s)
{
    if (s->run.empty()) return QSLC_OK;
    std::vector<GateOp> gates;
    gates.swap(s->run);
    const uint64_t mask = s->run_mask;
    run_drop(s);
    if (gates.size() == 1 || group_mode() != GROUP_RUNS || s->n < 4 || !run_pays(s, gates))
        return launch_each(s, gates);
    return s->dtype == QSLC_C128 ? launch_run<double>(s, gates, mask) : launch_run<float>(s, gates, mask);
}

int run_push(qslc_state *s, const GateOp &g)
{
    const GroupMode mode = group_mode();
    const bool pairs = mode == GROUP_PAIRS || (mode == GROUP_RUNS && !is_move(g.code) && !runs_any(s));
    bool fits = true;
    if (!s->run.empty()) {
        if (pairs) fits = !is_two_qubit(g.code) && !is_two_qubit(s->run[0].code) && s->run[0].q1 != g.q1;
        else {
            const Shape sh = shape_of(s);
            const uint64_t high = (s->run_mask | qubits_of(g)) >> sh.low;
            fits = unsigned(__builtin_popcountll(high)) <= sh.bits - sh.low &&
                   s->run_ops + lowered_of(g.code) <= RUN_MAX_GATES &&
                   (runs_any(s) || is_move(s->run[0].code));
        }
    }
    if (!fits) {
        const int rc = run_release(s);
        if (rc) return rc;
    }
    s->run.push_back(g);
    s->run_mask |= qubits_of(g);
    s->run_ops += lowered_of(g.code);
    if (mode == GROUP_OFF || (pairs && (is_two_qubit(g.code) || s->run.size() == 2))) return run_release(s);
    return QSLC_OK;
}

int run_bounds_error() { return unit_bounds_error(); }

void run_drop(qslc_state *s)
{
    s->run.clear();
    s->run_mask = 0;
    s->run_ops = 0;
}

}  // namespace qslc
