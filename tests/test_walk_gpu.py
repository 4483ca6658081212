"""The device walk of sequential sums (seqsum.cuh) against the oracle, on
states that leave its common path: sums below and above the size from which
tiles are only sampled, mass in one corner (so the samples mislead), zero
tiles, equal terms (rounding ties), terms that fall by a factor each (every
binade crossed, subnormals at the end), one term above all others, and
complex64 sums that stall."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(rng, n, dtype):
    dim = 1 << n
    dense = rng.normal(size=dim) + 1j * rng.normal(size=dim)
    out = {"dense": dense}
    corner = dense.copy()
    corner[dim // 8:] *= 1e-9
    out["corner"] = corner
    late = np.zeros(dim, dtype=complex)
    late[dim - max(dim // 16, 1):] = dense[dim - max(dim // 16, 1):]
    out["late"] = late
    out["equal"] = np.ones(dim, dtype=complex)
    ties = np.ones(dim, dtype=complex)
    ties[0] = 2.0 ** 12
    out["ties"] = ties
    out["falling"] = 2.0 ** (-np.arange(dim, dtype=float) / (dim / 600 if dtype == np.complex128 else dim / 80)) + 0j
    peak = dense * 1e-3
    peak[dim // 3] = 40
    out["peak"] = peak
    return {k: (v / np.linalg.norm(v)).astype(dtype) for k, v in out.items()}


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [2, 12, 14, 19, 23])
def test_walked_sums_and_shots_match_oracle(qsl, port, n, dtype):
    rng = np.random.default_rng(n)
    u = rng.random(300)
    u[0], u[1] = 0.0, np.nextafter(1.0, 0.0)
    if dtype == np.complex64:
        u = np.minimum(u.astype(np.float32), np.float32(1 - 2.0 ** -24)).astype(np.float64)
    for name, st in states(rng, n, dtype).items():
        gpu, cpu = qsl.Qubits(n, state=st, dtype=dtype), port.PortQubits(n, state=st, fp32=dtype == np.complex64)
        for q, o in ((0, 0), (n - 1, 1), (n // 2, 0)):
            assert gpu.prob(q, o) == cpu.prob(q, o), (name, q, o)
        assert np.array_equal(gpu.sample_shots(u), cpu.sample_all(u)), name


@pytest.mark.parametrize("n", [6, 13, 18])
def test_terms_with_and_without_easy_squares(qsl, port, n):
    # |a|^2 on the integer pipes takes parts with exponent fields 512 to 1533 and a low bit set; a warp
    # with any other part takes the FP64 pipe.  Whole stretches of each kind, and single parts among easy ones.
    rng = np.random.default_rng(n)
    dim = 1 << n
    st = rng.normal(size=dim) + 1j * rng.normal(size=dim)
    st /= np.linalg.norm(st)
    v = st.view(np.float64)
    odd = np.array([0.0, -0.0, 2.0 ** -511, np.nextafter(2.0 ** -511, 0), 2.0 ** -512, 1e-200, 5e-324, 2.0 ** -5, 1.5 * 2.0 ** -9,
                    1 + 2.0 ** -26, 2.0 ** -7 * (1 + 2.0 ** -25)])
    odd[-2:] *= 2.0 ** -6
    few = rng.random(v.size) < 0.02
    v[few] = rng.choice(odd, few.sum())
    v[v.size // 4: v.size // 4 + v.size // 8] = rng.choice(odd[:7], v.size // 8)
    u = rng.random(200)
    gpu, cpu = qsl.Qubits(n, state=st), port.PortQubits(n, state=st)
    for q in range(0, n, 3):
        for o in (0, 1):
            assert gpu.prob(q, o) == cpu.prob(q, o), (q, o)
    assert np.array_equal(gpu.sample_shots(u), cpu.sample_all(u))
