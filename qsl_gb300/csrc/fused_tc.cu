// fused_tc.cu -- five-qubit dense blocks on the 5th-generation tensor cores.
//
// A fused block U (32 x 32 complex) applied to every group of 32 amplitudes
// is the matrix product D = A * B^T with
//   A [groups x 64]  one row per group: its amplitudes as (re, im) pairs,
//   B [64 x 64]      the real form of U: B[2o+c][2v+d] from U[o][v],
//   D [groups x 64]  the new amplitudes, (re, im) pairs again.
// A CTA takes 128 groups per tile (M = 128), N = 64, K = 64, and issues
// tcgen05.mma kind::tf32 from one thread with the fp32 accumulator in
// tensor memory.  FP32 accuracy comes from the 3xTF32 split: every operand
// x = hi + lo with hi, lo TF32, and D = A_hi B_hi + A_hi B_lo + A_lo B_hi
// (the A_lo B_lo term is below FP32 resolution).
//
// A lives in tensor memory (row i in lane i, one 32-bit column per K entry):
// a thread's group is its lane's row, so the split goes there straight from
// registers.  From shared memory, writing the two halves of A and reading
// them twice for the MMAs took more than half of the SM's 128 bytes a clock,
// and the tiles left 34 KB of L1 for loads in flight: 3.44 ms a block of a
// 30-qubit state (5.0 TB/s) against 2.61 ms (6.6 TB/s) now, of which 0.54 ms
// come from loading two tiles ahead instead of one.
//
// B uses the canonical K-major shared-memory layout without swizzle: core
// matrices of 8 rows x 16 bytes, 128 contiguous bytes each, ordered K-chunk
// fastest then 8-row group; the descriptors' leading byte offset is the step
// between K-adjacent core matrices (128 B) and the stride byte offset the step
// between 8-row groups (K/4 * 128 B).
//
// Every wait is bounded: if the MMA completion never arrives the kernel
// records an error code, releases its tensor memory and returns.
#include "qslc_internal.cuh"

#include <cstring>
#include <vector>

namespace qslc {
namespace {

constexpr int TC_M = 128;   // groups per tile
constexpr int TC_N = 64;
constexpr int TC_K = 64;
constexpr int CORE_BYTES = 128;
constexpr int B_BYTES = TC_N * TC_K * 4;     // 16 KB per split half
// Tensor memory of a CTA: A_hi, A_lo and D, one 32-bit column per K or N.
constexpr uint32_t TMEM_COLS = 256, TM_HI = 0, TM_LO = TC_K, TM_D = 2 * TC_K;
constexpr int ROW_BYTES = 8 * 32 + 16;       // a group's amplitudes in shared memory; 16 bytes keep rows apart
constexpr int TILE_BYTES = TC_M * ROW_BYTES;
constexpr long long WAIT_LIMIT = 1ll << 26;

__device__ __forceinline__ uint32_t core_offset(int row, int k)
{
    return uint32_t(((row >> 3) * (TC_K / 4) + (k >> 2)) * CORE_BYTES + (row & 7) * 16 + (k & 3) * 4);
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr)
{
    const uint32_t lbo = CORE_BYTES, sbo = (TC_K / 4) * CORE_BYTES;
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFF);
    d |= uint64_t((lbo >> 4) & 0x3FFF) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFF) << 32;
    d |= uint64_t(1) << 46;                  // descriptor version of sm_100 tcgen05
    return d;                                // base offset 0, no swizzle
}

// kind::tf32 instruction descriptor: D f32, A/B tf32, both K-major, N, M
constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(TC_N >> 3) << 17) |
                           (uint32_t(TC_M >> 4) << 24);

__device__ __forceinline__ uint32_t to_tf32(float x)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15};\n" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}

// A from tensor memory (row i in lane i, column k its K entry k), B from shared memory
__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t acc)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(IDESC), "r"(acc)
        : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase)
{
    uint32_t done = 0;
    for (long long it = 0; it < WAIT_LIMIT && !done; it++) {
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(phase));
    }
    return done != 0;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// bmat: B_hi then B_lo, each [64 n][64 k] row-major fp32 (tf32 values).
//
// Pipeline per tile: the 32 amplitudes of this thread's group are in registers;
// they are split into tensor memory, one thread issues the MMAs, and every
// thread at once loads the tile after the next into the same registers, so two
// tiles are on their way at any time.  Tiles cover disjoint groups, so reading
// ahead of the stores is safe.
//
// LOW is for blocks with three or four of the lowest four qubits, whose
// groups lie so close that a warp's access to one amplitude of each takes 32
// sectors in up to 32 lines: the tile's 4096 amplitudes are copied to shared
// memory and back in ascending order of their place in memory instead, 256
// bytes a warp at worst in pieces of 32.  Blocks of a 29-qubit state, us,
// direct and LOW: qubits 0-4 4214 and 1970, {0, 1, 2, 10, 11} 2590 and 2121, 1-5
// 2385 and 2095, {0, 1, 10, 11, 12} 1838 and 2114, 2-6 1667 and 2102, 10-14 1378
// and 2132.
template <bool LOW>
__global__ void __launch_bounds__(TC_M) k_dense_tc(float2 *__restrict__ st, uint64_t ngroups,
                                                   const float *__restrict__ bmat, uint4 pos_lo,
                                                   unsigned pos_hi, int *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *b_hi = smem, *b_lo = b_hi + B_BYTES;
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int arrived;
    __shared__ uint64_t s_off[32], s_copy[32];
    __shared__ uint32_t s_row[32];
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned pos[5] = {pos_lo.x, pos_lo.y, pos_lo.z, pos_lo.w, pos_hi};
    if (tid < 32) {
        uint64_t o = 0;
#pragma unroll
        for (int j = 0; j < 5; j++)
            if (tid & (1 << j)) o |= uint64_t(1) << pos[j];
        s_off[tid] = o;
    }
    // B into the canonical layout (rows n, columns k)
    for (int i = tid; i < TC_N * TC_K; i += TC_M) {
        const int n = i / TC_K, k = i % TC_K;
        const uint32_t o = core_offset(n, k);
        *reinterpret_cast<float *>(b_hi + o) = bmat[i];
        *reinterpret_cast<float *>(b_lo + o) = bmat[TC_N * TC_K + i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const uint32_t mbar_s = uint32_t(__cvta_generic_to_shared(&mbar));
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_s));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    if (warp == 0) {
        const uint32_t slot = uint32_t(__cvta_generic_to_shared(&tmem_slot));
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;
    const uint32_t b_hi_s = uint32_t(__cvta_generic_to_shared(b_hi));
    const uint32_t b_lo_s = uint32_t(__cvta_generic_to_shared(b_lo));
    const uint64_t ntiles = ngroups / TC_M;
    auto group_base = [&](uint64_t t, int row) {
        uint64_t b = t * TC_M + row;
#pragma unroll
        for (int j = 0; j < 5; j++) b = insert0(b, pos[j]);
        return b;
    };
    const uint64_t step = gridDim.x;
    auto load = [&](float2 (&a)[32], uint64_t t) {
        if (t >= ntiles) return;
        const uint64_t b = group_base(t, tid);
#pragma unroll
        for (int v = 0; v < 32; v++) a[v] = st[b | s_off[v]];
    };
    // LOW: the tile as TC_M rows in shared memory, two tiles by turns.  Copy i
    // of a thread is local amplitude 128 i + tid; a tile's 12 bits, ascending,
    // are each a bit of the row or of the place in it.
    unsigned char *const rows = smem + 2 * B_BYTES;
    uint64_t my_off = 0;
    uint32_t my_row = 0;
    if constexpr (LOW) {
        auto place = [&](unsigned l, uint64_t &g, uint32_t &r) {
            unsigned q = 0, nv = 0, nr = 0;
            g = 0;
            r = 0;
            for (int j = 0; j < 12; j++, q++) {
                while (nr == 7 && q != pos[nv]) q++;         // 7 row bits found: only the block's are left
                const bool block = nv < 5 && q == pos[nv];
                if ((l >> j) & 1) {
                    g |= uint64_t(1) << q;
                    r += block ? 8u << nv : uint32_t(ROW_BYTES) << nr;
                }
                if (block) nv++;
                else nr++;
            }
        };
        place(unsigned(tid), my_off, my_row);
        if (tid < 32) place(unsigned(tid) << 7, s_copy[tid], s_row[tid]);
        __syncthreads();
    }
    auto copy_in = [&](uint64_t t, int half) {
        if (t < ntiles) {
            const float2 *src = st + (group_base(t, 0) | my_off);
            const uint32_t dst = uint32_t(__cvta_generic_to_shared(rows + half * TILE_BYTES)) + my_row;
#pragma unroll 8
            for (int i = 0; i < 32; i++)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + s_row[i]), "l"(src + s_copy[i])
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t lanes = tmem + (uint32_t(warp * 32) << 16);   // this warp's rows
    uint32_t phase = 0;
    // one tile, whose amplitudes are in `a` (LOW: on their way to rows);
    // false when the wait ran out
    auto tile = [&](float2 (&a)[32], uint64_t t, int half) -> bool {
        unsigned char *const buf = rows + half * TILE_BYTES;
        if constexpr (LOW) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float4 x = *reinterpret_cast<const float4 *>(buf + tid * ROW_BYTES + 16 * j);
                a[2 * j] = make_float2(x.x, x.y);
                a[2 * j + 1] = make_float2(x.z, x.w);
            }
        }
        const uint64_t base = LOW ? group_base(t, 0) : group_base(t, tid);
        // row `tid` of A: K entries 2v, 2v + 1 are amplitude v's (re, im)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float x = i & 1 ? a[8 * c + i / 2].y : a[8 * c + i / 2].x;
                hi[i] = to_tf32(x);
                lo[i] = to_tf32(x - __uint_as_float(hi[i]));
            }
            tmem_st16(lanes + TM_HI + uint32_t(16 * c), hi);
            tmem_st16(lanes + TM_LO + uint32_t(16 * c), lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0) {
            uint32_t acc = 0;
#pragma unroll
            for (int s = 0; s < TC_K / 8; s++) {       // K = 8 per instruction: two core matrices
                const uint32_t koff = uint32_t(2 * s * CORE_BYTES);
                const uint64_t bh = smem_desc(b_hi_s + koff), bl = smem_desc(b_lo_s + koff);
                mma_tf32(tmem + TM_D, tmem + TM_HI + 8 * s, bh, acc);
                acc = 1;
                mma_tf32(tmem + TM_D, tmem + TM_HI + 8 * s, bl, 1);
                mma_tf32(tmem + TM_D, tmem + TM_LO + 8 * s, bh, 1);
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                mbar_s));
        }
        // the amplitudes of the tile after the next travel from here on
        if constexpr (!LOW) load(a, t + 2 * step);
        // one thread polls the barrier (bounded); the block follows its outcome
        if (tid == 0) arrived = mbar_wait(mbar_s, phase) ? 1 : 0;
        __syncthreads();
        if (!arrived) {
            if (tid == 0) {
                atomicExch(err, 1);
                mbar_wait(mbar_s, phase);            // give work in flight a last bounded wait
            }
            return false;
        }
        phase ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;");
        // row tid of D: lane tid of tensor memory, 64 fp32 columns
#pragma unroll
        for (int c = 0; c < 4; c++) {
            uint32_t r[16];
            tmem_ld16(lanes + TM_D + uint32_t(16 * c), r);
            asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int v = 8 * c + i;
                const float2 x = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                if constexpr (LOW) *reinterpret_cast<float2 *>(buf + tid * ROW_BYTES + 8 * v) = x;
                else st[base | s_off[v]] = x;
            }
        }
        if constexpr (LOW) {
            __syncthreads();
#pragma unroll 8
            for (int i = 0; i < 32; i++)
                st[(base | my_off) + s_copy[i]] = *reinterpret_cast<const float2 *>(buf + my_row + s_row[i]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if constexpr (LOW) copy_in(t + 2 * step, half);
        return true;
    };
    float2 a0[32], a1[32];
    if constexpr (LOW) {
        copy_in(blockIdx.x, 0);
        copy_in(blockIdx.x + step, 1);
    } else {
        load(a0, blockIdx.x);
        load(a1, blockIdx.x + step);
    }
    for (uint64_t t = blockIdx.x; t < ntiles; t += 2 * step) {
        if (!tile(a0, t, 0)) break;
        if (t + step >= ntiles || !tile(LOW ? a0 : a1, t + step, 1)) break;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// host: TF32 rounding, to nearest with ties away from zero (cvt.rna)
float tf32_host(float x)
{
    uint32_t b;
    std::memcpy(&b, &x, 4);
    if ((b & 0x7F800000u) != 0x7F800000u) b = (b + 0x1000u) & ~0x1FFFu;
    float r;
    std::memcpy(&r, &b, 4);
    return r;
}

}  // namespace

// B = real form of the 32x32 complex block U (U[o*32+v]), split hi/lo.
void tc_pack_block(const std::vector<cd> &U, float *out)
{
    float *hi = out, *lo = out + TC_N * TC_K;
    for (int o = 0; o < 32; o++)
        for (int v = 0; v < 32; v++) {
            const double ur = U[size_t(o) * 32 + v].real(), ui = U[size_t(o) * 32 + v].imag();
            const double val[2][2] = {{ur, -ui}, {ui, ur}};   // [c_out][c_in]
            for (int co = 0; co < 2; co++)
                for (int ci = 0; ci < 2; ci++) {
                    const float x = float(val[co][ci]);
                    const float h = tf32_host(x);
                    const float l = tf32_host(x - h);
                    const int idx = (2 * o + co) * TC_K + (2 * v + ci);
                    hi[idx] = h;
                    lo[idx] = l;
                }
        }
}

size_t tc_block_floats() { return size_t(2) * TC_N * TC_K; }

bool tc_usable(const qslc_state *s) { return s->n >= 12; }

int tc_launch(qslc_state *s, const float *d_b, const unsigned *pos, int *d_err)
{
    const uint64_t ngroups = uint64_t(1) << (s->n - 5);
    const uint64_t tiles = ngroups / TC_M;
    const unsigned grid = unsigned(std::min<uint64_t>(tiles, uint64_t(sm_count()) * 2));
    auto go = [&](auto *kern, int smem) -> int {
        QSLC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kern<<<grid, TC_M, smem, s->stream>>>(static_cast<float2 *>(s->amps), ngroups, d_b,
                                              make_uint4(pos[0], pos[1], pos[2], pos[3]), pos[4], d_err);
        return QSLC_OK;
    };
    const bool low = pos[2] < 4;          // three of the lowest four (positions ascend)
    const int rc = low ? go(k_dense_tc<true>, 2 * B_BYTES + 2 * TILE_BYTES) : go(k_dense_tc<false>, 2 * B_BYTES);
    if (rc) return rc;
    s->launches++;
    QSLC_CUDA(cudaGetLastError());
    return QSLC_OK;
}

}  // namespace qslc
