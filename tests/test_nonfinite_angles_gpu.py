"""Angles that are infinite or NaN: the sine and cosine are NaN, and so is every
amplitude that the gate writes, a zero too (0 * NaN).  From |0...0>, where
nearly all amplitudes are zeros, each form that applies a gate -- two gates to a
sweep, runs, a gate's own sweep, number-preserving and resizeable states, the
batching form -- leaves NaNs where the oracle does, and its bits elsewhere."""
import numpy as np
import pytest

from conftest import random_np_state

pytestmark = pytest.mark.gpu

ANGLES = [np.inf, -np.inf, np.nan]
ANGLED1 = ("rotateX", "rotateY", "rotateZ", "phase")
ANGLED2 = ("controlRotateX", "controlRotateY", "controlRotateZ", "controlPhase", "npRotateX", "npRotateY")


def same(a, b):
    real = np.float64 if a.dtype == np.complex128 else np.float32
    a, b = np.ascontiguousarray(a).view(real), np.ascontiguousarray(b).view(real)
    nan = np.isnan(b)
    raw = np.uint64 if real == np.float64 else np.uint32
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a.view(raw)[~nan], b.view(raw)[~nan])


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [10, 19, 20])
def test_held_gates(qsl, port, n, dtype):
    """20 qubits: complex128 pairs (k_group2); below, runs (k_run)."""
    for i, name in enumerate(ANGLED1 + ANGLED2):
        angle = ANGLES[i % 3]
        two = name in ANGLED2
        # controls that are set, and a target in and outside a warp
        circ = [("pauliX", 1, None, 0.0), ("pauliX", n - 1, None, 0.0), ("rotateX", 2, None, 0.3),
                (name, 1, n - 2, angle) if two else (name, n - 2 if i & 1 else 3, None, angle)]
        if not two:
            circ.append(("hadamard", 0, None, 0.0))
        for flush in (False, True):
            gpu, cpu = qsl.Qubits(n, dtype=dtype), port.PortQubits(n, fp32=dtype == np.complex64)
            for g in circ:
                gpu.gate(*g)
                if flush:
                    gpu.flush()
                cpu.gate(*g)
            got = gpu.getState()
            assert np.isnan(cpu.state).any()
            assert same(got, cpu.state), (name, angle, flush)


@pytest.mark.parametrize("angle", ANGLES)
def test_number_preserving_gates(qsl, port, angle):
    n, w = 9, 4
    st = random_np_state(np.random.default_rng(5), n, w)
    st[np.flatnonzero(st)[1:]] = 0
    for name in ("rotateZ", "phase", "controlRotateZ", "controlPhase", "npRotateX", "npRotateY"):
        q2 = None if name in ("rotateZ", "phase") else 6
        gpu, cpu = qsl.QubitsNP(state=st), port.PortNPQubits(n, w, state=st)
        gpu.gate(name, 2, q2, angle)
        cpu.gate(name, 2, q2, angle)
        assert same(gpu.getState(), cpu.state), name


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_batch(qsl, port, dtype):
    """Instances below a tile and above it (14 and 15 qubits); the last
    layer's last rotateZ has the angle, or one in the middle."""
    ns = np.array([2, 6, 11, 13, 14, 15], dtype=np.uint32)
    ls = np.full(ns.size, 2, dtype=np.uint32)
    fp32 = dtype == np.complex64
    b = qsl.Batch(ns, ls, 0, dtype=dtype)
    rng = np.random.default_rng(3)
    # two basis states: rotateY angles of 0 leave zeros, one qubit is turned
    angles, at = np.zeros(b.angle_count), 0
    for i, n in enumerate(ns):
        a = angles[at:at + 4 * int(n)].reshape(2, int(n), 2)
        a[0, 0, 0] = rng.uniform(0.3, 1.0)
        a[:, :, 1] = rng.uniform(0, 3, (2, int(n)))
        a[1, int(n) - 1, 1] = ANGLES[i % 3]
        at += 4 * int(n)
    if fp32:
        angles = angles.astype(np.float32).astype(np.float64)
    probs, _ = b.run(angles, np.zeros(0))
    at = 0
    for i, n in enumerate(int(x) for x in ns):
        sim = port.PortQubits(n, fp32=fp32)
        a = angles[at:at + 4 * n].reshape(2, n, 2)
        at += 4 * n
        for l in range(2):
            for k, name in enumerate(("rotateY", "rotateZ")):
                for q in range(n):
                    sim.gate(name, q, None, a[l, q, k])
            for q in range(n - 1):
                sim.gate("controlNot", q, q + 1)
        want = np.array([[sim.prob(q, 0), sim.prob(q, 1)] for q in range(n)])
        assert np.isnan(want).all()
        assert np.array_equal(np.isnan(probs[i]), np.isnan(want)), n
