// gateops.cuh -- one-qubit updates chosen at run time, for the sweep that
// applies two gates (gates.cu k_group2).
//
// `op` is a PairOp, or GROUP_DIAG + a DiagOp for phase and pauliZ (which act
// on the members with the bit set).
#pragma once

#include "gatemath.cuh"

namespace qslc {

constexpr int GROUP_DIAG = 16;

template <class T, int OP>
__device__ __forceinline__ void group_pair(cplx<T> &a0, cplx<T> &a1, const Coef<T> &k)
{
    if constexpr (sizeof(T) == 8 && OP != P_SWAP && OP != P_Y) pair_either<OP>(a0, a1, k, slow_coef(k), &k.kd);
    else pair_update<T, OP>(a0, a1, k);
}
template <class T>
__device__ __forceinline__ void group_phase(cplx<T> &a, const Coef<T> &k)
{
    if constexpr (sizeof(T) == 8) {
        phase_either<false>(a, k, slow_coef(k));
    } else {
        diag_update<T, D_PHASE>(a, k);
    }
}

// One gate on the pairs (x0, x1) and (y0, y1); x1 and y1 are the members
// with the gate's bit set.  ARITH false: only the gates that move amplitudes
// or change signs.
template <class T, bool ARITH>
__device__ __forceinline__ void group_apply(int op, cplx<T> &x0, cplx<T> &x1, cplx<T> &y0, cplx<T> &y1,
                                            const Coef<T> &k)
{
    if constexpr (!ARITH) {
        if (op == P_SWAP) {
            pair_update<T, P_SWAP>(x0, x1, k);
            pair_update<T, P_SWAP>(y0, y1, k);
        } else if (op == P_Y) {
            pair_update<T, P_Y>(x0, x1, k);
            pair_update<T, P_Y>(y0, y1, k);
        } else {
            diag_update<T, D_NEG>(x1, k);
            diag_update<T, D_NEG>(y1, k);
        }
        return;
    }
    switch (op) {
    case P_SWAP:
        group_pair<T, P_SWAP>(x0, x1, k);
        group_pair<T, P_SWAP>(y0, y1, k);
        break;
    case P_Y:
        group_pair<T, P_Y>(x0, x1, k);
        group_pair<T, P_Y>(y0, y1, k);
        break;
    case P_H:
        group_pair<T, P_H>(x0, x1, k);
        group_pair<T, P_H>(y0, y1, k);
        break;
    case P_RX:
        group_pair<T, P_RX>(x0, x1, k);
        group_pair<T, P_RX>(y0, y1, k);
        break;
    case P_RY:
        group_pair<T, P_RY>(x0, x1, k);
        group_pair<T, P_RY>(y0, y1, k);
        break;
    case P_RZ:
        group_pair<T, P_RZ>(x0, x1, k);
        group_pair<T, P_RZ>(y0, y1, k);
        break;
    case GROUP_DIAG + D_NEG:
        diag_update<T, D_NEG>(x1, k);
        diag_update<T, D_NEG>(y1, k);
        break;
    default:                                  // GROUP_DIAG + D_PHASE
        group_phase<T>(x1, k);
        group_phase<T>(y1, k);
        break;
    }
}

}  // namespace qslc
