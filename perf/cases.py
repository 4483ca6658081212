"""The work that users of this framework have it do, as timed cases.

Every case goes through the public Python API (``Qubits``, ``QubitsNP``,
``QubitsResize``, ``Batch``), as a program that imports ``qsl_gb300`` does.
Sizes follow the framework's benchmark configurations (10 to 20 qubits from
|0...0>, 28 qubits of Hamming weight 14, 30 qubits dense, batches of 10 to 20
qubits) and their neighbours.  Kinds of case:

``circuit``  layers of one-qubit gates on every qubit and two-qubit gates on
             a random pairing; from |0...0> or on a dense state; complex128
             or complex64; with ``fuse`` set, in the fused precision form.
``gates``    one call of each of the 21 gates, on random qubits of a dense state.
``measure``  mid-circuit measurement: a prepared state is assigned to a working
             one, some qubits' probabilities read, shots sampled, some qubits
             measured (and so collapsed).
``np``       number-preserving gates on a dense state of fixed Hamming weight.
``resize``   rounds of parity checks: append an ancilla, controlNots into it,
             measure it out.
``batch``    many small ansatz circuits with probabilities and shots, on host
             arrays.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qsl_gb300 as qsl
from qsl_gb300 import workloads

DTYPES = {"c128": np.complex128, "c64": np.complex64}
ROTATIONS = ("rotateX", "rotateY", "rotateZ")


def listed():
    return [
        # a small variational circuit: every call is short, launches and host calls count
        {"name": "circuit_c128_10q", "kind": "circuit", "n": 10, "layers": 8, "mix": "cnot", "dtype": "c128",
         "start": "zero", "fuse": 0},
        # the 20-qubit benchmark circuit from |0...0>: the state stays in L2
        {"name": "circuit_c128_20q", "kind": "circuit", "n": 20, "layers": 20, "mix": "cnot", "dtype": "c128",
         "start": "zero", "fuse": 0},
        # layers of the 30-qubit benchmark circuit in its dense middle: 16 GiB in HBM
        {"name": "circuit_c128_30q", "kind": "circuit", "n": 30, "layers": 2, "mix": "mixed", "dtype": "c128",
         "start": "dense", "fuse": 0},
        # single precision at an odd size
        {"name": "circuit_c64_25q", "kind": "circuit", "n": 25, "layers": 4, "mix": "mixed", "dtype": "c64",
         "start": "dense", "fuse": 0},
        # every gate of the API once: controlled and number-preserving forms too
        {"name": "gates_c128_27q", "kind": "gates", "n": 27, "rounds": 1, "dtype": "c128"},
        # the 20-qubit benchmark's measurements: all probabilities, 10,000 shots
        {"name": "measure_c128_20q", "kind": "measure", "n": 20, "probs": 20, "measures": 2, "shots": 10000,
         "dtype": "c128"},
        # the large benchmark's measurements: 8 measured qubits, 100,000 shots
        {"name": "measure_c128_28q", "kind": "measure", "n": 28, "probs": 2, "measures": 8, "shots": 100000,
         "dtype": "c128"},
        # the number-preserving benchmark's state and gate mix
        {"name": "np_c128_28q_w14", "kind": "np", "n": 28, "w": 14, "gates": 200, "dtype": "c128"},
        # repeated parity checks with an ancilla that comes and goes
        {"name": "resize_c128_23q", "kind": "resize", "n": 23, "rounds": 4, "dtype": "c128"},
        # the precision form: gate runs fused into five-qubit blocks on the tensor cores
        {"name": "fused_c64_30q", "kind": "circuit", "n": 30, "layers": 4, "mix": "mixed", "dtype": "c64",
         "start": "dense", "fuse": 5},
        # the batching benchmark in single precision, whole
        {"name": "batch_c64_4096", "kind": "batch", "inst": 4096, "nmin": 10, "nmax": 20, "lmin": 4, "lmax": 16,
         "shots": 1024, "dtype": "c64"},
        # a quarter of it in double precision
        {"name": "batch_c128_1024", "kind": "batch", "inst": 1024, "nmin": 10, "nmax": 20, "lmin": 4, "lmax": 16,
         "shots": 1024, "dtype": "c128"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "gates", "measure", "np", "resize", "batch"])
    dtype = rng.choice(["c128", "c128", "c64"])
    if kind == "circuit":
        n = rng.randint(5, 30)            # the state spans 2^5 to 2^30 amplitudes
        most = 40 if n < 16 else 16 if n < 22 else 6 if n < 27 else 2
        fuse = rng.choice([0, 4, 5]) if dtype == "c64" else 0
        return {"kind": "circuit", "n": n, "layers": rng.randint(1, most), "mix": rng.choice(["cnot", "mixed"]),
                "dtype": dtype, "start": rng.choice(["zero", "dense"]) if n < 24 else "dense", "fuse": fuse}
    if kind == "gates":
        n = rng.randint(3, 29)
        return {"kind": "gates", "n": n, "rounds": rng.randint(1, 3), "dtype": dtype}
    if kind == "measure":
        n = rng.randint(6, 28)
        return {"kind": "measure", "n": n, "probs": rng.randint(1, min(n, 12)), "measures": rng.randint(1, min(n, 8)),
                "shots": _log_int(rng, 1, 100000), "dtype": dtype}
    if kind == "np":
        n = rng.randint(8, 28)
        return {"kind": "np", "n": n, "w": rng.randint(1, n - 1), "gates": rng.randint(20, 200), "dtype": dtype}
    if kind == "resize":
        return {"kind": "resize", "n": rng.randint(5, 25), "rounds": rng.randint(1, 6), "dtype": dtype}
    nmin = rng.randint(6, 11)
    nmax = rng.randint(nmin, 20)
    return {"kind": "batch", "inst": _log_int(rng, 32, 1024), "nmin": nmin, "nmax": nmax,
            "lmin": rng.randint(1, 4), "lmax": rng.randint(4, 16), "shots": _log_int(rng, 16, 1024), "dtype": dtype}


# ---- what a program has in hand before the call -----------------------------

def _circuit(case, seed):
    make = workloads.layered_cnot if case["mix"] == "cnot" else workloads.layered_mixed
    return make(case["n"], case["layers"], seed)


def _all_gates(case, seed):
    rng = np.random.default_rng(seed)
    n, circ = case["n"], []
    for _ in range(case["rounds"]):
        for g in list(qsl.GATE1) + list(qsl.GATE2):
            a = float(rng.uniform(0, 2 * np.pi)) if g in qsl.ANGLED else 0.0
            q = [int(x) for x in rng.choice(n, 2, replace=False)]
            circ.append((g, q[0], q[1] if g in qsl.GATE2 else None, a))
    return circ


def _parity_checks(case, seed):
    """Per round: the data qubits checked and the uniform its measurement draws."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    return [([int(x) for x in rng.choice(n, min(4, n), replace=False)], float(rng.random()))
            for _ in range(case["rounds"])]


def _dense(count, seed, out=None, dtype=torch.float64):
    """`count` Gaussian amplitudes as {re, im} rows, of norm 1."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    v = out if out is not None else torch.empty((count, 2), dtype=dtype, device="cuda")
    v.normal_(generator=g)
    v.mul_(1.0 / float(torch.linalg.vector_norm(v.view(-1), dtype=torch.float64)))
    return v


def _measurement(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    return {"probs": [int(x) for x in rng.choice(n, case["probs"], replace=False)],
            "measures": [(int(x), float(rng.random())) for x in rng.choice(n, case["measures"], replace=False)],
            "uniforms": workloads.uniforms(case["shots"], seed)}


def _batch(case, seed):
    # the instances' sizes are the program's, and the same for every run of a case
    rng = np.random.default_rng(case["inst"])
    ns = rng.integers(case["nmin"], case["nmax"] + 1, case["inst"]).astype(np.uint32)
    ls = rng.integers(case["lmin"], case["lmax"] + 1, case["inst"]).astype(np.uint32)
    rng = np.random.default_rng(seed)
    angles = rng.uniform(0, 2 * np.pi, int(np.sum(2 * ns.astype(np.int64) * ls)))
    return ns, ls, angles, workloads.uniforms(case["inst"] * case["shots"], seed)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        ns, ls, s["angles"], s["uniforms"] = _batch(case, seed)
        s["batch"] = qsl.Batch(ns, ls, case["shots"], dtype=DTYPES[case["dtype"]])
        return s
    dt = DTYPES[case["dtype"]]
    if kind == "np":
        q = qsl.QubitsNP(case["n"], nones=case["w"], dtype=dt)
        s["circuit"] = workloads.np_mix(case["n"], case["gates"], seed)
    elif kind == "resize":
        q = qsl.QubitsResize(case["n"], dtype=dt)
        s["checks"] = _parity_checks(case, seed)
    else:
        q = qsl.Qubits(case["n"], dtype=dt)
        if kind == "measure":
            s["what"] = _measurement(case, seed)
        else:
            s["circuit"] = _circuit(case, seed) if kind == "circuit" else _all_gates(case, seed)
    q.synchronize()
    view = q.device_view()
    if case.get("start") != "zero":
        _dense(view.shape[0], seed, out=view)
        torch.cuda.synchronize()
    s["q"], s["view"] = q, view
    if case.get("fuse"):
        q.set_fusion(case["fuse"])
    if kind in ("measure", "resize"):
        s["work"] = q.copy()
        s["work"].synchronize()
        if kind == "measure":
            s["workview"] = s["work"].device_view()
    return s


# ---- one pass ---------------------------------------------------------------

SMALL = 12   # states of up to this many qubits are read back to the host, as a small program does


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        probs, shots = s["batch"].run(s["angles"], s["uniforms"])
        return {"probs": np.concatenate([p.reshape(-1) for p in probs]), "shots": shots.view(np.int64)}
    q = s["q"]
    if kind == "measure":
        w, what = s["work"], s["what"]
        w.assign(q)
        p = np.array([w.prob(t, 0) for t in what["probs"]])
        shots = w.sample_shots(what["uniforms"])
        out = np.array([w.measure(t, u) for t, u in what["measures"]])
        return {"probs": p, "shots": shots.view(np.int64), "outcomes": out, "state": s["workview"]}
    if kind == "resize":
        w, out = s["work"], []
        w.assign(q)
        for data, u in s["checks"]:
            w.appendQubit()
            for d in data:
                w.controlNot(d, w.nqubits - 1)
            out.append(w.measureOut(w.nqubits - 1, u))
        return {"outcomes": np.array(out), "state": w.device_view()}
    if case.get("start") == "zero":
        q.reset()
    workloads.apply(q, s["circuit"])
    if case["n"] <= SMALL and kind == "circuit":
        return q.getState()
    q.flush()
    return s["view"]


# ---- what a pass cannot do without ------------------------------------------

def _gate_flops(name, dim):
    """Floating-point operations of one gate in the reference's formulas: 12 for a rotated pair, 8 for
    a Hadamard pair, 6 for a phased amplitude."""
    if name in ("hadamard",):
        return 4 * dim
    if name in ROTATIONS:
        return 6 * dim
    if name == "phase":
        return 3 * dim
    if name in ("controlRotateX", "controlRotateY", "controlRotateZ", "npRotateX", "npRotateY"):
        return 3 * dim
    if name in ("controlHadamard", "npHadamard"):
        return 2 * dim
    if name == "controlPhase":
        return 1.5 * dim
    return 0


def work(case):
    kind = case["kind"]
    amp = 16 if case["dtype"] == "c128" else 8
    if kind == "batch":
        ns, ls, _, _ = _batch(case, 0)
        ns, ls = ns.astype(np.float64), ls.astype(np.float64)
        dim = 2.0 ** ns
        flops = float(np.sum(dim * (ls * ns * 12 + 3 + ns)))
        host = float(np.sum(2 * ns * ls * 8) + case["inst"] * case["shots"] * 16 + np.sum(2 * ns * 8))
        return {"bytes": host, "flops": flops}
    if kind == "np":
        dim = math.comb(case["n"], case["w"])
        per = {g: _gate_flops(g, dim) for g in ("npRotateX", "swap", "phase", "controlPhase")}
        return {"bytes": 2 * amp * dim, "flops": case["gates"] * sum(per.values()) / 4}
    dim = 1 << case["n"]
    if kind == "measure":
        # the state copied, each probability's half read, the CDF's terms, each measurement's half and its collapse
        reads = 0.5 * case["probs"] + 1 + 0.5 * case["measures"]
        return {"bytes": amp * dim * (2 + reads + 1.5 * case["measures"]) + 16 * case["shots"],
                "flops": dim * (4 * reads + case["measures"])}
    if kind == "resize":
        return {"bytes": 2 * amp * dim, "flops": case["rounds"] * dim * 5}
    circ = _circuit(case, 0) if kind == "circuit" else _all_gates(case, 0)
    return {"bytes": 2 * amp * dim, "flops": float(sum(_gate_flops(g, dim) for g, _, _, _ in circ))}


# ---- the same in 64 bits, in plain torch ------------------------------------

def _bit(v, n, q):
    """`v` (rows of 2^n amplitudes) as (rows, high, bit q, low)."""
    return v.view(v.shape[0], 1 << (n - 1 - q), 2, 1 << q)


def _mix(a0, a1, m):
    """(a0, a1) <- m (a0, a1) in place; m: four numbers or tensors that broadcast."""
    if m[1] is None:                       # diagonal
        if m[0] is not None:
            a0.mul_(m[0])
        a1.mul_(m[3])
        return
    t0 = a0 * m[0] + a1 * m[1]
    a1.mul_(m[3]).add_(a0 * m[2])
    a0.copy_(t0)


def _matrix(g, a):
    c, s = math.cos(a / 2), math.sin(a / 2)
    r = 1 / math.sqrt(2)
    return {"pauliX": (0, 1, 1, 0), "pauliY": (0, -1j, 1j, 0), "pauliZ": (None, None, None, -1),
            "hadamard": (r, r, r, -r), "phase": (None, None, None, complex(math.cos(a), math.sin(a))),
            "rotateX": (c, -1j * s, -1j * s, c), "rotateY": (c, -s, s, c),
            "rotateZ": (complex(c, -s), None, None, complex(c, s))}[g]


CONTROLLED = {"controlNot": "pauliX", "controlY": "pauliY", "controlZ": "pauliZ", "controlRotateX": "rotateX",
              "controlRotateY": "rotateY", "controlRotateZ": "rotateZ", "controlPhase": "phase",
              "controlHadamard": "hadamard"}
EXCHANGE = {"swap": "pauliX", "fswap": "pauliX", "npRotateX": "rotateX", "npRotateY": "rotateY",
            "npHadamard": "hadamard"}


def _apply_exact(v, n, circ):
    for g, q1, q2, a in circ:
        if q2 is None:
            x = _bit(v, n, q1)
            _mix(x[:, :, 0], x[:, :, 1], _matrix(g, a))
            continue
        lo, hi = min(q1, q2), max(q1, q2)
        x = v.view(v.shape[0], 1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)

        def part(b1, b2):
            bh, bl = (b1, b2) if q1 == hi else (b2, b1)
            return x[:, :, bh, :, bl]
        if g in CONTROLLED:
            _mix(part(1, 0), part(1, 1), _matrix(CONTROLLED[g], a))
        else:
            _mix(part(1, 0), part(0, 1), _matrix(EXCHANGE[g], a))
            if g == "fswap":
                part(1, 1).neg_()
    return v


def _start(case, seed, count):
    """The state that prepare() makes, in complex128."""
    if case.get("start") == "zero":
        v = torch.zeros(1, count, dtype=torch.complex128, device="cuda")
        v[0, 0] = 1
        return v
    dt = torch.float64 if case["dtype"] == "c128" else torch.float32
    return torch.view_as_complex(_dense(count, seed, dtype=dt).to(torch.float64)).view(1, count)


def _out(v):
    return torch.view_as_real(v.view(-1))


def _weight_index(n, w):
    i = torch.arange(1 << n, dtype=torch.int64, device="cuda")
    c = torch.zeros(1 << n, dtype=torch.int8, device="cuda")
    for q in range(n):
        c += ((i >> q) & 1).to(torch.int8)
    return torch.nonzero(c == w).view(-1)


def _exact_batch(case, seed):
    ns, ls, angles, _ = _batch(case, seed)
    at = np.concatenate([[0], np.cumsum(2 * ns.astype(np.int64) * ls)])
    probs = [None] * len(ns)
    groups = {}
    for i, key in enumerate(zip(ns.tolist(), ls.tolist())):
        groups.setdefault(key, []).append(i)
    for (n, layers), members in groups.items():
        for k in range(0, len(members), 64):
            ids = members[k:k + 64]
            ang = torch.tensor(np.stack([angles[at[i]:at[i + 1]] for i in ids])).view(len(ids), layers, n, 2).cuda() / 2
            c, s = ang.cos().to(torch.complex128), ang.sin().to(torch.complex128)
            v = torch.zeros(len(ids), 1 << n, dtype=torch.complex128, device="cuda")
            v[:, 0] = 1
            for l in range(layers):
                for q in range(n):
                    cq, sq = c[:, l, q, 0].view(-1, 1, 1), s[:, l, q, 0].view(-1, 1, 1)
                    x = _bit(v, n, q)
                    _mix(x[:, :, 0], x[:, :, 1], (cq, -sq, sq, cq))
                for q in range(n):
                    cq, sq = c[:, l, q, 1].view(-1, 1, 1), s[:, l, q, 1].view(-1, 1, 1)
                    x = _bit(v, n, q)
                    _mix(x[:, :, 0], x[:, :, 1], (cq - 1j * sq, None, None, cq + 1j * sq))
                for q in range(n - 1):
                    _apply_exact(v, n, [("controlNot", q, q + 1, 0.0)])
            p = v.real.square() + v.imag.square()
            both = torch.stack([_bit(p, n, q).sum(dim=(1, 3)) for q in range(n)], 1).cpu().numpy()
            for j, i in enumerate(ids):
                probs[i] = both[j].reshape(-1)
    return {"probs": np.concatenate(probs), "shots": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    n = case["n"]
    if kind == "np":
        idx = _weight_index(n, case["w"])
        full = torch.zeros(1, 1 << n, dtype=torch.complex128, device="cuda")
        full[0, idx] = _start(case, seed, idx.numel())[0]
        _apply_exact(full, n, workloads.np_mix(n, case["gates"], seed))
        return _out(full[0, idx])
    v = _start(case, seed, 1 << n)
    if kind == "circuit" or kind == "gates":
        _apply_exact(v, n, _circuit(case, seed) if kind == "circuit" else _all_gates(case, seed))
        if kind == "circuit" and n <= SMALL:
            # getState's complex array, as {re, im} values
            return v.view(-1).cpu().numpy()
        return _out(v)

    def prob0(q):
        x = torch.view_as_real(_bit(v, n, q)[:, :, 0].contiguous())
        return float(x.square().sum())

    def collapse(q, u):
        p0 = prob0(q)
        o = 0 if u < p0 else 1
        x = _bit(v, n, q)
        x[:, :, o].mul_(1 / math.sqrt(p0 if o == 0 else 1 - p0))
        x[:, :, 1 - o].zero_()
        return o
    if kind == "measure":
        what = _measurement(case, seed)
        p = np.array([prob0(t) for t in what["probs"]])
        for t, u in what["measures"]:
            collapse(t, u)
        return {"probs": p, "shots": None, "outcomes": None, "state": _out(v)}
    for data, u in _parity_checks(case, seed):
        v = torch.cat([v, torch.zeros_like(v)], 1)
        n += 1
        _apply_exact(v, n, [("controlNot", d, n - 1, 0.0) for d in data])
        o = collapse(n - 1, u)
        v = _bit(v, n, n - 1)[:, 0, o].contiguous()
        n -= 1
    return {"outcomes": None, "state": _out(v)}
