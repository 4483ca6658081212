"""Runs of gates in one sweep (run.cu) give the bits of the gates one by one,
for every gate, at the sizes around the tiles (one tile, two, many; the
threads of a CTA not filled), with qubits inside and outside the tile, on
dense states and on states of zeros, infinities' neighbours and subnormals.
Applying the held gate after each call (flush) sends each through its own
sweep, which is the reference here; complex128 is also held to the oracle."""
import numpy as np
import pytest

from conftest import bits, random_state

pytestmark = pytest.mark.gpu

ONE = ("pauliX", "pauliY", "pauliZ", "hadamard", "phase", "rotateX", "rotateY", "rotateZ")
TWO = ("controlNot", "controlY", "controlZ", "controlRotateX", "controlRotateY", "controlRotateZ", "controlPhase",
       "controlHadamard", "swap", "fswap", "npRotateX", "npRotateY", "npHadamard")


def gates(rng, n, count, names=ONE + TWO):
    out = []
    for _ in range(count):
        g = str(rng.choice(names))
        q = [int(x) for x in rng.choice(n, 2, replace=False)]
        out.append((g, q[0], q[1] if g in TWO else None, float(rng.uniform(0, 2 * np.pi))))
    return out


def run(qsl, st, circ, one_by_one):
    sim = qsl.Qubits(state=st, dtype=st.dtype)
    for g in circ:
        sim.gate(*g)
        if one_by_one:
            sim.flush()
    return sim.getState(), sim.launches()


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [2, 4, 5, 8, 9, 10, 11, 13, 15, 18, 20, 21])
def test_runs_give_the_bits_of_single_sweeps(qsl, n, dtype):
    rng = np.random.default_rng(n)
    st = random_state(rng, n, dtype)
    circ = gates(rng, n, 150)
    a, held = run(qsl, st, circ, False)
    b, alone = run(qsl, st, circ, True)
    assert np.array_equal(bits(a), bits(b))
    if n >= 4:
        assert held < alone


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [6, 12, 19])
def test_runs_on_states_of_odd_values(qsl, n, dtype):
    rng = np.random.default_rng(100 + n)
    real = np.float64 if dtype == np.complex128 else np.float32
    tiny = float(np.finfo(real).tiny)
    odd = np.array([0.0, -0.0, tiny, -tiny / 8, 1.0, -0.5, 1.5, float(np.finfo(real).max) / 8, 1e-31], dtype=real)
    for share in (0.01, 0.6):
        st = random_state(rng, n, dtype)
        v = st.view(real)
        at = rng.random(v.size) < share
        v[at] = rng.choice(odd, int(at.sum()))
        circ = gates(rng, n, 12)
        a, _ = run(qsl, st, circ, False)
        b, _ = run(qsl, st, circ, True)
        # a NaN (of an infinity times zero) is a NaN in both; its payload is the instruction's own
        x, y = a.view(real), b.view(real)
        assert np.array_equal(np.isnan(x), np.isnan(y))
        assert np.array_equal(np.nan_to_num(x, nan=0.0).view(np.uint8), np.nan_to_num(y, nan=0.0).view(np.uint8))


@pytest.mark.parametrize("n", [10, 13, 18])
def test_runs_from_the_zero_state_match_the_oracle(qsl, port, n):
    rng = np.random.default_rng(200 + n)
    circ = gates(rng, n, 60)
    gpu, cpu = qsl.Qubits(n), port.PortQubits(n)
    for g in circ:
        gpu.gate(*g)
        cpu.gate(*g)
    assert np.array_equal(bits(gpu.getState()), bits(cpu.state))


@pytest.mark.parametrize("n", [18, 24])
def test_runs_of_moves_on_large_states(qsl, n):
    """Two-qubit moves, signs and phases between pairs of one-qubit gates."""
    rng = np.random.default_rng(300 + n)
    moves = ("controlNot", "controlY", "controlZ", "controlPhase", "swap", "fswap")
    circ = []
    for _ in range(3):
        circ += gates(rng, n, 3, ONE) + gates(rng, n, 9, moves)
    st = random_state(rng, n)
    a, held = run(qsl, st, circ, False)
    b, alone = run(qsl, st, circ, True)
    assert np.array_equal(bits(a), bits(b))
    assert held < alone


@pytest.mark.parametrize("n, dtype", [(n, np.complex128) for n in (7, 12, 17, 19)] + [(n, np.complex64) for n in (7, 12, 14)])
def test_runs_around_the_small_register_form(qsl, n, dtype):
    # complex128 states of at most 19 qubits and complex64 ones of at most 13 keep fewer amplitudes a thread
    rng = np.random.default_rng(300 + n)
    st = random_state(rng, n, dtype)
    circ = gates(rng, n, 120)
    a, held = run(qsl, st, circ, False)
    b, alone = run(qsl, st, circ, True)
    assert np.array_equal(bits(a), bits(b))
    assert held < alone
