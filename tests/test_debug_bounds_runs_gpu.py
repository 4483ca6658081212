"""The debug build's index checks (-DQSLC_DEBUG_BOUNDS) in each way that gates
are held: runs (k_run), pairs (k_group2) and not at all, complex128 and
complex64.  A debug library gives the default build's bits and reports nothing.
One that checks against half the state (=2) skips the upper half's items and
reports them, so every form has its checks; nothing is read or written outside
the state."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import bits, random_state

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, {root!r})
import qsl_gb300 as q
q.lib({lib!r})
d = np.load({inp!r})
for i, part in enumerate({parts!r}):
    sim = q.Qubits(state=d["state"], dtype=d["state"].dtype)
    for k in part:
        b = int(d["q2"][k])
        sim.gate(str(d["names"][k]), int(d["q1"][k]), None if b < 0 else b, float(d["ang"][k]))
    try:
        np.save({out!r} % i, sim.getState())
        print("taken")
    except q.LogicError as e:
        print("refused:", e)
"""


@pytest.fixture(scope="module")
def libraries(tmp_path_factory):
    from qsl_gb300 import build as b
    b.build()
    work = tmp_path_factory.mktemp("debug")
    out, objs, jobs = {"default": b.LIB}, {}, []
    others = [os.path.join(b.OBJ, f) for f in sorted(os.listdir(b.OBJ))
              if f.endswith(".o") and f not in ("gates.o", "run.o")]
    for tag, value in (("debug", 1), ("half", 2)):
        objs[tag] = [str(work / f"{unit}_{tag}.o") for unit in ("gates", "run")]
        for unit, obj in zip(("gates", "run"), objs[tag]):
            jobs.append(subprocess.Popen([b.nvcc(), *b.ARCH, *b.NVCC_FLAGS, f"-DQSLC_DEBUG_BOUNDS={value}", "-c",
                                          os.path.join(b.CSRC, unit + ".cu"), "-o", obj]))
    assert [j.wait() for j in jobs] == [0] * len(jobs)
    cudalib = os.path.join(os.path.dirname(os.path.dirname(b.nvcc())), "lib64")
    for tag in objs:
        out[tag] = str(work / f"libqslc_{tag}.so")
        r = subprocess.run([b.nvcc(), *b.ARCH, "-shared", "-o", out[tag], *others, *objs[tag], "-lcudart", "-lpthread",
                            "-L", cudalib, "-Xlinker", "-rpath", "-Xlinker", cudalib], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return out


def applied(tmp_path, lib, group, st, circ, parts):
    """What became of each part (indices into circ), on a fresh copy of st."""
    inp, out = str(tmp_path / "in.npz"), str(tmp_path / "out%d.npy")
    names, q1, q2, ang = (np.array(x) for x in zip(*circ))
    np.savez(inp, state=st, names=names, q1=q1, q2=q2, ang=ang)
    env = {k: v for k, v in os.environ.items() if not k.startswith("QSLC_")}
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, lib=lib, inp=inp, out=out, parts=parts)],
                       env=dict(env, QSLC_GROUP=group), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    said = r.stdout.splitlines()
    return [np.load(out % i) if x == "taken" else x for i, x in enumerate(said)]


ONE = ("hadamard", "phase", "rotateX", "rotateY", "pauliZ")
TWO = ("controlNot", "controlZ", "controlPhase", "controlRotateY", "swap", "fswap", "npRotateX")


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("group", ["", "1", "0"])
@pytest.mark.parametrize("n", [7, 14, 20])
def test_the_checks_pass_and_refuse(libraries, tmp_path, n, group, dtype):
    rng = np.random.default_rng(n)
    st = random_state(rng, n, dtype)
    circ = []
    for _ in range(5):
        for g in ONE + TWO:
            a, b = (int(x) for x in rng.choice(n, 2, replace=False))
            circ.append((g, a, b if g in TWO else -1, float(rng.uniform(0, 2 * np.pi))))
    whole = [list(range(len(circ)))]
    a, = applied(tmp_path, libraries["default"], group, st, circ, whole)
    b, = applied(tmp_path, libraries["debug"], group, st, circ, whole)
    assert isinstance(b, np.ndarray) and np.array_equal(bits(a), bits(b))
    # each gate alone, two together, a run: the upper half is refused
    parts = [[k] for k in range(len(ONE + TWO))] + [[0, 1], whole[0][:12]]
    said = applied(tmp_path, libraries["half"], group, st, circ, parts)
    assert len(said) == len(parts)
    for part, out in zip(parts, said):
        assert isinstance(out, str) and out.startswith("refused:"), (group, part)
        assert 1 << (n - 1) <= int(out.rsplit(" ", 1)[1]) < 1 << n
