"""Warps that leave the easy arithmetic (lean.cuh) for the general update:
states whose amplitudes mix ordinary values with zeros, subnormals, values of
few significant bits and values at both ends of the exponent range, one such
operand in a warp, in many, or in all; and gate constants the easy products
refuse (a cosine of exactly 1, a tiny sine).  The results are the oracle's
bits."""
import numpy as np
import pytest

from conftest import bits, random_np_state, random_state

pytestmark = pytest.mark.gpu

ODD = [0.0, -0.0, 5e-324, 1e-310, 2.3e-308, 1.5 * 2.0 ** -700, 3.0 * 2.0 ** -959, 1.5, -0.75, 1.0, 2.0 ** 1000,
       -1.1 * 2.0 ** 1021, 2.0 ** -957, 1.1 * 2.0 ** -958]
PLAIN = [("hadamard", 1), ("rotateX", 1), ("rotateY", 1), ("rotateZ", 1), ("phase", 1), ("controlRotateX", 2),
         ("controlRotateY", 2), ("controlRotateZ", 2), ("controlPhase", 2), ("controlHadamard", 2),
         ("npRotateX", 2), ("npRotateY", 2), ("npHadamard", 2)]
NP = [("rotateZ", 1), ("phase", 1), ("controlPhase", 2), ("controlRotateZ", 2), ("npRotateX", 2), ("npRotateY", 2),
      ("npHadamard", 2)]
ANGLES = [0.7, 2.9, 1e-9, 2.0 ** -80, np.pi]


def spoil(rng, st, share):
    """Put odd values in `share` of the real and imaginary parts."""
    v = st.view(np.float64)
    at = rng.random(v.size) < share
    v[at] = rng.choice(ODD, int(at.sum()))
    return st


@pytest.mark.parametrize("n", [2, 6, 11])
@pytest.mark.parametrize("share", [0.002, 0.1, 0.7])
def test_odd_operands_give_the_oracles_bits(qsl, port, n, share):
    rng = np.random.default_rng(n + int(1000 * share))
    for name, k in PLAIN:
        for angle in ANGLES:
            st = spoil(rng, random_state(rng, n), share)
            q = [int(x) for x in rng.choice(n, 2, replace=False)]
            gpu, cpu = qsl.Qubits(n, state=st), port.PortQubits(n, state=st)
            for sim in (gpu, cpu):
                sim.gate(name, q[0], q[1] if k == 2 else None, angle)
            assert np.array_equal(bits(gpu.getState()), bits(cpu.state)), (name, angle, q)


@pytest.mark.parametrize("share", [0.002, 0.3])
def test_odd_operands_in_grouped_sweeps(qsl, port, share):
    rng = np.random.default_rng(int(1000 * share))
    n = 10
    for first in ("hadamard", "rotateX", "rotateY", "rotateZ", "phase"):
        for second in ("hadamard", "rotateX", "phase"):
            st = spoil(rng, random_state(rng, n), share)
            q = [int(x) for x in rng.choice(n, 2, replace=False)]
            gpu, cpu = qsl.Qubits(n, state=st), port.PortQubits(n, state=st)
            for sim in (gpu, cpu):
                sim.gate(first, q[0], None, 1.3)
                sim.gate(second, q[1], None, 0.4)
            # an infinity from the largest values may become a NaN, whose payload is the machine's own
            a, b = gpu.getState().view(np.float64), cpu.state.view(np.float64)
            assert np.array_equal(np.isnan(a), np.isnan(b))
            a, b = np.nan_to_num(a, nan=0.0), np.nan_to_num(b, nan=0.0)
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (first, second, q)


@pytest.mark.parametrize("share", [0.01, 0.5])
def test_odd_operands_in_number_preserving_sweeps(qsl, port, share):
    rng = np.random.default_rng(int(1000 * share))
    n, w = 11, 5
    base = random_np_state(rng, n, w)
    keep = base != 0
    for name, k in NP:
        for angle in ANGLES:
            st = base.copy()
            part = spoil(rng, st[keep], share)
            part[0] = 0.5                        # the weight stays readable from the state
            st[keep] = part
            q = [int(x) for x in rng.choice(n, 2, replace=False)]
            gpu, cpu = qsl.QubitsNP(n, nones=w), port.PortNPQubits(n, w, state=st)
            gpu.setState(st)
            for sim in (gpu, cpu):
                sim.gate(name, q[0], q[1] if k == 2 else None, angle)
            assert np.array_equal(bits(gpu.getState()), bits(cpu.state)), (name, angle, q)
