"""Runs on states above 31 qubits, whose indices take 64 bits (k_run's wide form):
32 qubits in complex64.  Gates on six qubits, the lowest and the highest among
them, from |0...0>: the 64 amplitudes they reach are the bits of the same circuit
on six qubits, and every other one stays zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, AT = 32, (0, 3, 11, 20, 30, 31)
ONE = ("pauliX", "pauliY", "pauliZ", "hadamard", "phase", "rotateX", "rotateY", "rotateZ")
TWO = ("controlNot", "controlY", "controlZ", "controlRotateX", "controlRotateY", "controlRotateZ", "controlPhase",
       "controlHadamard", "swap", "fswap", "npRotateX", "npRotateY", "npHadamard")


def test_runs_with_64_bit_indices(qsl, port):
    import torch
    rng = np.random.default_rng(32)
    gpu, cpu = qsl.Qubits(N, dtype=np.complex64), port.PortQubits(len(AT), fp32=True)
    gpu.synchronize()
    before = gpu.launches()
    circ = [("hadamard", q, None) for q in range(len(AT))]
    for _ in range(4):
        circ += [(str(g), int(rng.integers(len(AT))), None) for g in rng.permutation(ONE)]
        circ += [(str(g), *(int(x) for x in rng.choice(len(AT), 2, replace=False))) for g in rng.permutation(TWO)]
    for g, a, b in circ:
        x = float(rng.uniform(0, 2 * np.pi))
        gpu.gate(g, AT[a], None if b is None else AT[b], x)
        cpu.gate(g, a, b, x)
    gpu.synchronize()
    assert gpu.launches() - before < len(circ) / 4           # runs, not sweeps
    view = gpu.device_view()
    index = [sum(((i >> k) & 1) << q for k, q in enumerate(AT)) for i in range(1 << len(AT))]
    got = view[torch.tensor(index, device="cuda")].cpu().numpy().view(np.complex64).reshape(-1)
    assert np.array_equal(got.view(np.uint32), cpu.state.view(np.uint32))
    assert int(torch.count_nonzero(view)) == int(np.count_nonzero(got.view(np.float32)))
