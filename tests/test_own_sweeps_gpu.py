"""Every gate in a sweep of its own, complex128 and complex64: without held gates
(QSLC_GROUP=0), and with each switch that chooses the form of a gate's own sweep
(the splits QSLC_EMU_MASK*, staged sweeps QSLC_BULK, warp exchanges QSLC_SHFL).
One launch a gate shows that the sweeps named are the ones that ran; the bits are
the oracle's, for all gates, low and high qubits, ordinary angles and ones whose
sine or cosine is zero, tiny or of few bits.  QSLC_GROUP=1 beside a switch goes
on holding one-qubit gates in pairs."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import bits, random_state

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ONE = ("pauliX", "pauliY", "pauliZ", "hadamard", "phase", "rotateX", "rotateY", "rotateZ")
TWO = ("controlNot", "controlY", "controlZ", "controlRotateX", "controlRotateY", "controlRotateZ", "controlPhase",
       "controlHadamard", "swap", "fswap", "npRotateX", "npRotateY", "npHadamard")
EDGES = (0.0, np.pi / 2, np.pi, -np.pi, 2 * np.pi, 1e-30, 2.0 ** -70, 1e-10)

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, {root!r})
import qsl_gb300 as q
d = np.load({inp!r})
sim = q.Qubits(state=d["state"], dtype=d["state"].dtype)
sim.synchronize()
before = sim.launches()
for g, a, b, x in zip(d["names"], d["q1"], d["q2"], d["ang"]):
    sim.gate(str(g), int(a), None if int(b) < 0 else int(b), float(x))
sim.synchronize()
np.savez({out!r}, state=sim.getState(), launches=sim.launches() - before)
"""


def circuit(rng, n):
    circ = []
    for angle in list(rng.uniform(0, 2 * np.pi, 2)) + list(EDGES):
        for t in dict.fromkeys((0, 3, n - 1)):
            circ += [(g, t, -1, float(angle)) for g in rng.permutation(ONE)]
        for a, b in ((0, n - 1), (n - 1, 1), (2, 3)):
            circ += [(g, a, b, float(angle)) for g in rng.permutation(TWO)]
    return circ


def applied(tmp_path, env, st, circ):
    inp, out = str(tmp_path / "in.npz"), str(tmp_path / "out.npz")
    names, q1, q2, ang = (np.array(x) for x in zip(*circ))
    np.savez(inp, state=st, names=names, q1=q1, q2=q2, ang=ang)
    clean = {k: v for k, v in os.environ.items() if not k.startswith("QSLC_")}
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, inp=inp, out=out)],
                       env=dict(clean, **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    d = np.load(out)
    return d["state"], int(d["launches"])


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [4, 8, 12])
@pytest.mark.parametrize("env", [dict(QSLC_GROUP="0"), dict(QSLC_EMU_MASK="PPPQ,PPPQ,PPPF"),
                                 dict(QSLC_EMU_MASK_H="FEFE"), dict(QSLC_EMU_MASK_DIAG="PQ,QP,EF"),
                                 dict(QSLC_BULK="1"), dict(QSLC_SHFL="1"), dict(QSLC_SHFL="0")],
                         ids=lambda e: ",".join(f"{k}={v}" for k, v in e.items()))
def test_one_sweep_a_gate(qsl, port, tmp_path, env, n, dtype):
    rng = np.random.default_rng(n)
    st, circ = random_state(rng, n, dtype), circuit(rng, n)
    got, launches = applied(tmp_path, env, st, circ)
    assert launches == len(circ)
    cpu = port.PortQubits(n, fp32=dtype == np.complex64, state=st)
    for g, a, b, x in circ:
        cpu.gate(str(g), a, None if b < 0 else b, x)
    assert np.array_equal(bits(got), bits(cpu.state))


def test_pairs_when_asked_for(qsl, port, tmp_path):
    rng = np.random.default_rng(9)
    n = 8
    st = random_state(rng, n)
    circ = [("rotateX", t, -1, 0.3 + t) for t in range(n)]
    got, launches = applied(tmp_path, dict(QSLC_SHFL="1", QSLC_GROUP="1"), st, circ)
    assert launches == n // 2
    cpu = port.PortQubits(n, state=st)
    for g, a, b, x in circ:
        cpu.gate(g, a, None, x)
    assert np.array_equal(bits(got), bits(cpu.state))
