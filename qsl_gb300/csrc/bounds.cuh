// bounds.cuh -- index checks of the sweeps in debug builds.
//
// Debug builds (-DQSLC_DEBUG_BOUNDS) check each item's largest index
// against the state's size before the item is read or written: an index
// outside the state is recorded (the first one of a translation unit) and the
// item skipped, and the next call that reads the state returns QSLC_EINVAL with
// the index (debug_bounds_error).  The host validates every qubit index before
// a launch, so no call through the ABI should record one.
// -DQSLC_DEBUG_BOUNDS=2 checks against half the state, so that every sweep
// meets indices to refuse: a test of the checks, in which no access leaves the
// state either.  Default builds compile the checks to `true`.
#pragma once

#include "qslc_internal.cuh"

namespace qslc {

#ifdef QSLC_DEBUG_BOUNDS
static __device__ unsigned long long g_bad_index;   // first index outside a state, plus one; 0: none
__device__ __forceinline__ bool in_state_quiet(uint64_t i, uint64_t dim)
{
    return i < (dim >> (QSLC_DEBUG_BOUNDS - 1));
}
__device__ __forceinline__ bool in_state(uint64_t i, uint64_t dim)
{
    if (in_state_quiet(i, dim)) return true;
    atomicCAS(&g_bad_index, 0ull, (unsigned long long)i + 1ull);
    return false;
}
#define QSLC_IN_STATE(i, dim) ::qslc::in_state(uint64_t(i), uint64_t(dim))
#define QSLC_IN_STATE_QUIET(i, dim) ::qslc::in_state_quiet(uint64_t(i), uint64_t(dim))
#else
#define QSLC_IN_STATE(i, dim) true
#define QSLC_IN_STATE_QUIET(i, dim) true
#endif

// QSLC_EINVAL when a sweep of this translation unit met an index outside its
// state since the last call; QSLC_OK otherwise and in default builds.
static inline int unit_bounds_error()
{
#ifdef QSLC_DEBUG_BOUNDS
    unsigned long long bad = 0;
    QSLC_CUDA(cudaDeviceSynchronize());
    QSLC_CUDA(cudaMemcpyFromSymbol(&bad, g_bad_index, sizeof(bad)));
    if (bad) {
        const unsigned long long zero = 0;
        QSLC_CUDA(cudaMemcpyToSymbol(g_bad_index, &zero, sizeof(zero)));
        QSLC_CUDA(cudaDeviceSynchronize());
        return fail(QSLC_EINVAL, "a sweep indexed outside the state (debug bounds check): index " +
                                     std::to_string(bad - 1));
    }
#endif
    return QSLC_OK;
}

}  // namespace qslc
