"""The form of the gate arithmetic that takes zeros beside easy operands
(gatemath.cuh), and quarter turns, whose constants are powers of two: states whose
imaginary or real parts are zeros of either sign, all or some of them, half-empty
states, and states with odd values beside, through pairs (20 qubits), runs,
a gate's own sweep, number-preserving sweeps and the batching form.  The bits
are the oracle's."""
import numpy as np
import pytest

from conftest import bits, random_np_state, random_state

pytestmark = pytest.mark.gpu

ONE = ("hadamard", "rotateX", "rotateY", "rotateZ", "phase")
TWO = ("controlRotateX", "controlRotateY", "controlRotateZ", "controlPhase", "controlHadamard", "npRotateX", "npRotateY",
       "npHadamard")
ANGLES = (0.7, np.pi / 2, np.pi, -np.pi, 3 * np.pi, 2 * np.pi, 0.0)
KINDS = ("real", "imaginary", "minus", "parts", "half", "odd")


def state(rng, n, kind):
    st = random_state(rng, n)
    v = st.view(np.float64)
    if kind == "real":
        v[1::2] = 0.0
    elif kind == "imaginary":
        v[0::2] = -0.0
    elif kind == "minus":
        v[1::2] = np.where(rng.random(v.size // 2) < 0.5, 0.0, -0.0)
    elif kind == "half":
        st[rng.random(st.size) < 0.5] = 0
    else:
        at = rng.random(v.size) < 0.4
        v[at] = rng.choice([0.0, -0.0] + ([0.5, -1.0, 5e-324, 1e-310] if kind == "odd" else []), int(at.sum()))
    return st


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [5, 9, 20])
def test_held_and_single_gates(qsl, port, n, kind):
    rng = np.random.default_rng(n)
    for i, angle in enumerate(ANGLES if n < 20 else ANGLES[:3]):
        st = state(rng, n, kind)
        circ = [(str(g), int(rng.integers(n)), None, angle) for g in rng.permutation(ONE)]
        circ += [(circ[0][0], (circ[0][1] + 1) % n, None, angle), (circ[1][0], (circ[1][1] + 1) % n, None, 0.3)]
        for g in rng.permutation(TWO):
            a, b = (int(x) for x in rng.choice(n, 2, replace=False))
            circ.append((str(g), a, b, angle))
        cpu = port.PortQubits(n, state=st)
        for g in circ:
            cpu.gate(*g)
        for one_by_one in (False, True):
            gpu = qsl.Qubits(n, state=st)
            for g in circ:
                gpu.gate(*g)
                if one_by_one:
                    gpu.flush()
            assert np.array_equal(bits(gpu.getState()), bits(cpu.state)), (kind, angle, one_by_one)


@pytest.mark.parametrize("gate", ONE)
@pytest.mark.parametrize("kind", KINDS)
def test_pairs_of_one_gate(qsl, port, kind, gate):
    """Two gates of a kind and no more, on low and high qubits."""
    rng = np.random.default_rng(7)
    n = 20
    for a, b, angle in ((0, 1, 0.7), (3, 15, np.pi), (19, 4, np.pi / 2)):
        st = state(rng, n, kind)
        gpu, cpu = qsl.Qubits(n, state=st), port.PortQubits(n, state=st)
        for sim in (gpu, cpu):
            sim.gate(gate, a, None, angle)
            sim.gate(gate, b, None, angle)
        assert np.array_equal(bits(gpu.getState()), bits(cpu.state)), (a, b, angle)


@pytest.mark.parametrize("kind", KINDS)
def test_number_preserving_gates(qsl, port, kind):
    rng = np.random.default_rng(3)
    n, w = 11, 5
    base = random_np_state(rng, n, w)
    keep = base != 0
    for name in ("rotateZ", "phase", "controlPhase", "controlRotateZ", "npRotateX", "npRotateY", "npHadamard"):
        for angle in ANGLES:
            st = base.copy()
            part = state(rng, n, kind)[:int(keep.sum())].copy()
            part[0] = 0.5                        # the weight stays readable from the state
            st[keep] = part
            q = [int(x) for x in rng.choice(n, 2, replace=False)]
            gpu, cpu = qsl.QubitsNP(n, nones=w), port.PortNPQubits(n, w, state=st)
            gpu.setState(st)
            for sim in (gpu, cpu):
                sim.gate(name, q[0], q[1] if name.startswith(("control", "np")) else None, angle)
            assert np.array_equal(bits(gpu.getState()), bits(cpu.state)), (name, angle, q)


def test_batch_of_quarter_turns(qsl, port):
    """rotateY and rotateZ angles of 0, pi/2, pi and ordinary ones: real states, zeros and few-bit values."""
    rng = np.random.default_rng(12)
    ns, ls = np.array([2, 4, 9, 13, 14], dtype=np.uint32), np.array([3, 2, 3, 2, 2], dtype=np.uint32)
    b = qsl.Batch(ns, ls, 64)
    angles = rng.choice([0.0, np.pi / 2, np.pi, -np.pi, 1.1], b.angle_count)
    u = rng.random(ns.size * 64)
    probs, shots = b.run(angles, u)
    at = 0
    for i, (n, layers) in enumerate(zip(ns.tolist(), ls.tolist())):
        sim = port.PortQubits(n)
        a = angles[at:at + 2 * n * layers].reshape(layers, n, 2)
        at += 2 * n * layers
        for l in range(layers):
            for k, name in enumerate(("rotateY", "rotateZ")):
                for q in range(n):
                    sim.gate(name, q, None, a[l, q, k])
            for q in range(n - 1):
                sim.gate("controlNot", q, q + 1)
        want = np.array([[sim.prob(q, 0), sim.prob(q, 1)] for q in range(n)])
        assert np.array_equal(probs[i], want) and np.array_equal(shots[i], sim.sample_all(u[i * 64:(i + 1) * 64]))
