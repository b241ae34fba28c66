"""Timed cases of the state-vector engine: what its users call, over the sizes they call it at.

A case is a dict of plain values.  ``kind`` says which public entry point it goes through:

execute   ``device.LightningQubit.execute``: one evaluation of a variational circuit (reset, gates,
          Hamiltonian expectation value, probabilities of every wire), as an optimiser's loop
          does it on a small register, where launches and host work count.
gradient  ``device.LightningQubit.adjoint_jacobian``: Jacobian of a layered RX RY RZ + CNOT-ladder
          circuit with one PauliZ output (the plain configuration at 20 qubits, 600 parameters)
          or several outputs.
circuit   ``StateVector.apply_ops_fused``: 200 gates drawn from the gate sweep's kinds (one-wire
          gates, CNOT, CZ, SWAP, Toffoli, random two- and three-wire unitaries) on a live state.
gates     ``StateVector.apply`` / ``apply_matrix``: the same kinds one call at a time, the drop-in
          form of the C++ ``applyOperation`` / ``applyMatrix``.
matrix    ``StateVector.apply_matrix``: wide dense unitaries (block encodings, compiled blocks).
pauli     ``StateVector.expval_pauli``: a Hamiltonian of ZZ ring terms, X fields and
          Jordan-Wigner words, every word's value and the weighted sum.
sample    ``probs_device`` over every wire, a marginal, and shots from given uniforms.
batch     ``autograd.batched_expval``: one training step (forward and vector-Jacobian product) of
          many circuits at once: ``rot`` is general rotations + CNOT rings with a PauliZ output per
          qubit (the headline workload), ``hea`` the hardware-efficient ansatz of uneven widths
          and depths with a 3n-term Hamiltonian, ``grad`` says whether the gradient is taken.

Circuit structure (gates and wires) follows from the case; angles, matrices, states and weights
from the seed.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lightning-unification_b200"))

NP = {"c64": np.complex64, "c128": np.complex128}
AMP = {"c64": 8, "c128": 16}


def listed():
    return [
        # one objective evaluation on a small register: the smallest calls
        {"name": "execute 10q c128", "kind": "execute", "n": 10, "layers": 3, "dtype": "c128"},
        # a small odd-width gradient with several outputs
        {"name": "gradient 11q 3 outputs", "kind": "gradient", "n": 11, "layers": 4, "nobs": 3, "dtype": "c128"},
        # the plain configuration at its full size
        {"name": "gradient 20q c128", "kind": "gradient", "n": 20, "layers": 10, "nobs": 1, "dtype": "c128"},
        # deep circuits on wide states, in both precisions
        {"name": "circuit 26q c128", "kind": "circuit", "n": 26, "ngates": 200, "dtype": "c128"},
        {"name": "circuit 27q c64", "kind": "circuit", "n": 27, "ngates": 200, "dtype": "c64"},
        # gate by gate on a wide state
        {"name": "gates 28q c128", "kind": "gates", "n": 28, "ngates": 20, "dtype": "c128"},
        # dense blocks on four to six wires
        {"name": "matrix 25q c64", "kind": "matrix", "n": 25, "k0": 4, "k1": 6, "dtype": "c64"},
        # a chemistry-like Hamiltonian on a wide state
        {"name": "pauli 25q c128", "kind": "pauli", "n": 25, "words": 150, "dtype": "c128"},
        # readout of a wide state
        {"name": "sample 27q c64", "kind": "sample", "n": 27, "shots": 1000000, "dtype": "c64"},
        # the headline batch: a training step over 1024 circuits of 16 qubits
        {"name": "batch rot 16q c64", "kind": "batch", "circuit": "rot", "ncirc": 1024, "nmin": 16, "nmax": 16,
         "dmin": 8, "dmax": 8, "grad": True, "dtype": "c64"},
        # circuits of uneven width and depth, complex128
        {"name": "batch hea 10-18q c128", "kind": "batch", "circuit": "hea", "ncirc": 192, "nmin": 10, "nmax": 18,
         "dmin": 4, "dmax": 12, "grad": True, "dtype": "c128"},
        # many narrow circuits, values only (a parameter scan)
        {"name": "batch hea 8-12q c64", "kind": "batch", "circuit": "hea", "ncirc": 512, "nmin": 8, "nmax": 12,
         "dmin": 2, "dmax": 6, "grad": False, "dtype": "c64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds as listed, sizes over the ranges they stand for."""
    kind = rng.choice(["execute", "gradient", "gradient", "circuit", "circuit", "gates", "matrix", "pauli", "sample",
                       "batch", "batch", "batch"])
    dtype = rng.choice(["c64", "c128"])
    wide = 1 if dtype == "c64" else 0  # as many bytes: one more qubit in complex64
    if kind == "execute":
        return {"kind": kind, "n": rng.randint(4, 18), "layers": rng.randint(1, 8), "dtype": dtype}
    if kind == "gradient":
        n = rng.randint(5, 20)
        return {"kind": kind, "n": n, "layers": rng.randint(1, 8),
                "nobs": rng.choice([1, 1, 2, 3, min(n, 6)]), "dtype": dtype}
    if kind == "circuit":
        return {"kind": kind, "n": rng.randint(12, 26 + wide), "ngates": rng.randint(20, 200), "dtype": dtype}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(14, 27 + wide), "ngates": rng.randint(5, 20), "dtype": dtype}
    if kind == "matrix":
        k0 = rng.randint(3, 6)
        return {"kind": kind, "n": rng.randint(14, 24 + wide), "k0": k0, "k1": rng.randint(k0, 6), "dtype": dtype}
    if kind == "pauli":
        return {"kind": kind, "n": rng.randint(12, 25), "words": _log_int(rng, 8, 150), "dtype": dtype}
    if kind == "sample":
        return {"kind": kind, "n": rng.randint(12, 26 + wide), "shots": _log_int(rng, 1000, 1000000), "dtype": dtype}
    circuit = rng.choice(["rot", "hea"])
    if circuit == "rot":
        n = rng.randint(8, 16)
        return {"kind": kind, "circuit": circuit, "ncirc": _log_int(rng, 16, 400), "nmin": n, "nmax": n,
                "dmin": (d := rng.randint(2, 8)), "dmax": d, "grad": rng.random() < 0.7, "dtype": dtype}
    lo = rng.randint(6, 13)
    return {"kind": kind, "circuit": circuit, "ncirc": _log_int(rng, 16, 192), "nmin": lo,
            "nmax": lo + rng.randint(0, 4), "dmin": 2, "dmax": rng.randint(2, 10), "grad": rng.random() < 0.7,
            "dtype": dtype}


# ---- circuits: [(name, wires, angle slot or None, matrix slot or None)] --------------------------
def _fixed(case):
    """The generator of a case's structure: the same for every seed."""
    return random.Random(repr(sorted((k, v) for k, v in case.items() if k != "name")))


def _layered(n, layers):
    ops, p = [], 0
    for _ in range(layers):
        for q in range(n):
            for g in ("RX", "RY", "RZ"):
                ops.append((g, [q], p, None))
                p += 1
        for q in range(n - 1):
            ops.append(("CNOT", [q, q + 1], None, None))
    return ops, p


SWEEP = ("Hadamard", "RX", "RY", "RZ", "CNOT", "CZ", "SWAP", "Toffoli", "U2", "U3")
NWIRES = {"CNOT": 2, "CZ": 2, "SWAP": 2, "Toffoli": 3, "U2": 2, "U3": 3}


def _sweep(case):
    """Gates of the sweep's kinds in equal shares, in a shuffled order, on uniformly drawn wires."""
    r, n = _fixed(case), case["n"]
    kinds = [SWEEP[i % len(SWEEP)] for i in range(case["ngates"])]
    r.shuffle(kinds)
    ops, p, m = [], 0, []
    for kind in kinds:
        wires = r.sample(range(n), NWIRES.get(kind, 1))
        if kind in ("U2", "U3"):
            ops.append(("QubitUnitary", wires, None, len(m)))
            m.append(len(wires))
        elif kind in ("RX", "RY", "RZ"):
            ops.append((kind, wires, p, None))
            p += 1
        else:
            ops.append((kind, wires, None, None))
    return ops, p, m


def _blocks(case):
    """One dense matrix on each width k0..k1, wires drawn over the register."""
    r = _fixed(case)
    widths = list(range(case["k0"], case["k1"] + 1))
    return [("QubitUnitary", r.sample(range(case["n"]), k), None, i) for i, k in enumerate(widths)], 0, widths


def _words(case):
    """ZZ ring terms, X fields, and Jordan-Wigner words (X/Y on 1, 2 or 4 wires, Z between pairs)."""
    r, n, count = _fixed(case), case["n"], case["words"]
    words = [("ZZ", [q, (q + 1) % n]) for q in range(min(n, count // 3))]
    words += [("X", [q]) for q in range(min(n, count // 3))]
    while len(words) < count:
        ws = sorted(r.sample(range(n), r.choice([1, 2, 2, 4])))
        letters = {w: r.choice("XY") for w in ws}
        for lo, hi in zip(ws[0::2], ws[1::2]):
            for w in range(lo + 1, hi):
                letters[w] = "Z"
        wires = sorted(letters)
        words.append(("".join(letters[w] for w in wires), wires))
    return words


def _batch_shapes(case):
    """(qubits, layers) of every circuit."""
    r = _fixed(case)
    return [(r.randint(case["nmin"], case["nmax"]), r.randint(case["dmin"], case["dmax"]))
            for _ in range(case["ncirc"])]


def _batch_ops(circuit, n, layers):
    ops, p = [], 0
    for l in range(layers):
        for q in range(n):
            for g in (("RZ", "RY", "RZ") if circuit == "rot" else ("RY", "RZ")):
                ops.append((g, [q], p, None))
                p += 1
        step = (l % (n - 1)) + 1 if circuit == "rot" else 1
        for q in range(n):
            ops.append(("CNOT" if circuit == "rot" else "CZ", [q, (q + step) % n], None, None))
    return ops, p


def _batch_obs(circuit, n, coeffs):
    if circuit == "rot":
        return [[(1.0, "Z", [q])] for q in range(n)]
    words = [("ZZ", [q, (q + 1) % n]) for q in range(n)] + [("ZZ", [q, (q + 2) % n]) for q in range(n)]
    words += [("X", [q]) for q in range(n)]
    return [[(float(c), w, ws) for c, (w, ws) in zip(coeffs, words)]]


# ---- values from the seed ---------------------------------------------------------------------
def _unitaries(rng, widths):
    out = []
    for k in widths:
        z = rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k))
        q, r = np.linalg.qr(z)
        out.append(q * (np.diag(r) / np.abs(np.diag(r))))
    return out


def _state(case, seed):
    """A normalised Gaussian (Haar-like) state on the GPU in the case's precision."""
    g = torch.Generator(device="cuda").manual_seed(1000003 + seed)
    real = torch.float32 if case["dtype"] == "c64" else torch.float64
    x = torch.randn((1 << case["n"], 2), generator=g, device="cuda", dtype=real)
    x /= torch.linalg.vector_norm(x, dtype=torch.float64).to(real)
    return x


def _values(case, seed):
    """Everything the seed decides except the state: angles, matrices, coefficients, weights."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    v = {}
    if kind in ("execute", "gradient"):
        v["ops"], np_ = _layered(case["n"], case["layers"])
        v["angles"] = rng.uniform(0, 2 * np.pi, np_)
        v["coeffs"] = rng.normal(size=2 * case["n"])
    elif kind in ("circuit", "gates", "matrix"):
        v["ops"], np_, widths = _blocks(case) if kind == "matrix" else _sweep(case)
        v["angles"] = rng.uniform(0, 2 * np.pi, np_)
        v["mats"] = [m.astype(NP[case["dtype"]]) for m in _unitaries(rng, widths)]
    elif kind == "pauli":
        v["coeffs"] = rng.normal(size=case["words"])
    elif kind == "sample":
        v["uniforms"] = rng.random(case["shots"])
    else:
        shapes = _batch_shapes(case)
        per = 3 if case["circuit"] == "rot" else 2
        v["shapes"] = shapes
        v["angles"] = rng.uniform(0, 2 * np.pi, sum(per * n * d for n, d in shapes))
        v["coeffs"] = [rng.normal(size=3 * n) for n, _ in shapes]
        v["weights"] = rng.normal(size=sum(n if case["circuit"] == "rot" else 1 for n, _ in shapes))
    return v


class _DeviceArray:
    """A state's amplitudes as (2^n, 2) reals for torch, no copy."""

    def __init__(self, sv, dtype):
        self.sv = sv
        self.__cuda_array_interface__ = {"shape": (1 << sv.num_qubits, 2), "version": 3,
                                         "typestr": "<f4" if dtype == "c64" else "<f8",
                                         "data": (sv.device_ptr(), False)}


def _bound(v):
    """Operations as the C API binding takes them."""
    return [(name, wires, False, [] if p is None else [float(v["angles"][p])])
            + (() if m is None else (v["mats"][m],)) for name, wires, p, m in v["ops"]]


def prepare(case, seed):
    v = _values(case, seed)
    kind, dtype = case["kind"], NP[case["dtype"]]
    if kind in ("execute", "gradient"):
        from lightning_b200 import device as D
        n = case["n"]
        tape = [D.Operation(name, wires, [] if p is None else [float(v["angles"][p])]) for name, wires, p, _ in v["ops"]]
        if kind == "execute":
            obs = [D.tensor(D.named("PauliZ", q), D.named("PauliZ", (q + 1) % n)) for q in range(n)]
            obs += [D.named("PauliX", q) for q in range(n)]
            meas = [D.expval(D.hamiltonian(v["coeffs"], obs)), D.probs()]
        else:
            meas = [D.expval(D.named("PauliZ", q)) for q in range(case["nobs"])]
        return {"case": case, "dev": D.LightningQubit(n, c_dtype=dtype), "tape": D.Tape(tape, meas)}
    if kind in ("circuit", "gates", "matrix", "pauli", "sample"):
        from lightning_b200 import capi
        sv = capi.StateVector(case["n"], dtype)
        sv.set_stream(torch.cuda.current_stream().cuda_stream)
        view = torch.as_tensor(_DeviceArray(sv, case["dtype"]), device="cuda")
        view.copy_(_state(case, seed))
        s = {"case": case, "sv": sv, "view": view}
        if kind == "pauli":
            s.update(words=_words(case), coeffs=v["coeffs"])
        elif kind == "sample":
            s.update(probs=torch.empty(1 << case["n"], dtype=torch.float64, device="cuda"), uniforms=v["uniforms"])
        else:
            s.update(ops=_bound(v))
        return s
    from lightning_b200.batch import BatchedCircuits
    circuits, at = [], 0
    for (n, d), co in zip(v["shapes"], v["coeffs"]):
        ops, np_ = _batch_ops(case["circuit"], n, d)
        circuits.append({"num_qubits": n, "ops": [(g, w, False, []) for g, w, _, _ in ops],
                         "param_index": [-1 if p is None else at + p for _, _, p, _ in ops],
                         "observables": _batch_obs(case["circuit"], n, co)})
        at += np_
    return {"case": case, "engine": BatchedCircuits(circuits, at, dtype=dtype),
            "theta": torch.tensor(v["angles"], device="cuda", requires_grad=case["grad"]),
            "weights": torch.tensor(v["weights"], device="cuda")}


def run(s):
    kind = s["case"]["kind"]
    if kind == "execute":
        value, probs = s["dev"].execute(s["tape"])
        return [np.float64(value), probs]
    if kind == "gradient":
        return s["dev"].adjoint_jacobian(s["tape"])
    if kind == "circuit":
        s["sv"].apply_ops_fused(s["ops"])
        return s["view"]
    if kind in ("gates", "matrix"):
        for op in s["ops"]:
            if len(op) > 4:
                s["sv"].apply_matrix(op[4], op[1])
            else:
                s["sv"].apply(op[0], op[1], False, op[3])
        return s["view"]
    if kind == "pauli":
        values, total = s["sv"].expval_pauli(s["words"], s["coeffs"])
        return [values, np.float64(total)]
    if kind == "sample":
        sv = s["sv"]
        sv.probs_device(s["probs"].data_ptr())
        return [s["probs"], sv.probs(list(range(1, min(11, sv.num_qubits), 2))),
                sv.sample(len(s["uniforms"]), uniforms=s["uniforms"]).astype(np.int64)]
    from lightning_b200.autograd import batched_expval
    if not s["case"]["grad"]:
        return batched_expval(s["theta"], s["engine"])
    s["theta"].grad = None
    out = batched_expval(s["theta"], s["engine"])
    (out * s["weights"]).sum().backward()
    return [out.detach(), s["theta"].grad]


# ---- work ---------------------------------------------------------------------------------------
def _gate_flops(name, k):
    """Real operations per amplitude of the state."""
    if name == "QubitUnitary":
        return 8.0 * (1 << k)
    return {"Hadamard": 4.0, "RX": 6.0, "RY": 6.0, "RZ": 6.0, "CZ": 0.5}.get(name, 0.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        fl, by = 0.0, 0.0
        for n, d in _batch_shapes(case):
            ops, np_ = _batch_ops(case["circuit"], n, d)
            f = sum(_gate_flops(g, 1) for g, _, _, _ in ops) * (1 << n)
            nterms = n if case["circuit"] == "rot" else 3 * n
            f += 3.0 * nterms * (1 << n)
            if case["grad"]:  # the inverse on both states, one real inner product a parameter
                f += 2 * sum(_gate_flops(g, 1) for g, _, _, _ in ops) * (1 << n) + 4.0 * np_ * (1 << n)
            fl += f
            by += 8.0 * (np_ * (2 if case["grad"] else 1) + (n if case["circuit"] == "rot" else 1))
        return {"bytes": by, "flops": fl}
    n, N, S = case["n"], float(1 << case["n"]), AMP[case["dtype"]]
    if kind == "execute":
        ops, _ = _layered(n, case["layers"])
        return {"bytes": 8.0 * N, "flops": N * (sum(_gate_flops(g, 1) for g, _, _, _ in ops) + 6.0 * n)}
    if kind == "gradient":
        ops, np_ = _layered(n, case["layers"])
        f = sum(_gate_flops(g, 1) for g, _, _, _ in ops)
        return {"bytes": 8.0 * np_ * (1 + case["nobs"]), "flops": N * (f * (2 + case["nobs"]) + 4.0 * np_ * case["nobs"])}
    if kind in ("circuit", "matrix"):
        ops = (_blocks(case) if kind == "matrix" else _sweep(case))[0]
        passes = len(ops) if kind == "matrix" else 1
        return {"bytes": 2 * S * N * passes, "flops": N * sum(_gate_flops(g, len(w)) for g, w, _, _ in ops)}
    if kind == "gates":
        share = {"CNOT": 0.5, "SWAP": 0.5, "Toffoli": 0.25, "CZ": 0.25}
        ops = _sweep(case)[0]
        return {"bytes": 2 * S * N * sum(share.get(g, 1.0) for g, _, _, _ in ops),
                "flops": N * sum(_gate_flops(g, len(w)) for g, w, _, _ in ops)}
    if kind == "pauli":
        return {"bytes": S * N, "flops": 4.0 * N * case["words"]}
    return {"bytes": (S + 8.0) * N + 16.0 * case["shots"], "flops": 3.0 * N}


def tolerance(case):
    """What another order of the same operations at the same precision shows: about four times the
    distance measured from the 64-bit values."""
    kind, single = case["kind"], case["dtype"] == "c64"
    if kind in ("circuit", "gates", "matrix"):
        # up to 200 unitary steps on a normalised state (measured 6e-7, dense blocks 1.1e-6; 1.4e-15)
        return {"rel": 4e-6 if single else 1e-14}
    if kind == "sample":
        # FP64 reductions over the stored amplitudes in either precision; shots are whole numbers
        return {"rel": 1e-14, "max": 1e-13, "differ": 0.0}
    if kind == "pauli":
        # FP64 sums of 2^n products that largely cancel (a value is about 2^-n/2; measured 3e-14)
        return {"rel": 2e-13, "max": 2e-12}
    # values and gradients of whole circuits are differences about 2^-n/2 in size, so the amplitudes'
    # error counts for more the wider the state (measured 2e-6 at 16 qubits, 3e-15 at 20)
    return {"rel": (4e-5 if kind == "gradient" else 1e-5) if single else 1e-13}


# ---- the same in 64 bits, plain torch -------------------------------------------------------------
def _mat(name, t, dev="cuda"):
    """[B, d, d] (targets only) of a named gate at angles t [B]; controls are handled apart."""
    z, o = torch.zeros_like(t), torch.ones_like(t)
    c, s = torch.cos(t / 2), torch.sin(t / 2)
    cx = torch.complex
    if name == "RX":
        rows = [cx(c, z), cx(z, -s), cx(z, -s), cx(c, z)]
    elif name == "RY":
        rows = [cx(c, z), cx(-s, z), cx(s, z), cx(c, z)]
    elif name == "RZ":
        rows = [cx(c, -s), cx(z, z), cx(z, z), cx(c, s)]
    elif name == "Hadamard":
        r = math.sqrt(0.5)
        rows = [cx(r * o, z), cx(r * o, z), cx(r * o, z), cx(-r * o, z)]
    else:
        raise ValueError(name)
    return torch.stack(rows, -1).reshape(-1, 2, 2)


def _const(name):
    m = {"CNOT": (4, [(2, 3)]), "SWAP": (4, [(1, 2)]), "Toffoli": (8, [(6, 7)])}
    if name == "CZ":
        return np.diag([1, 1, 1, -1]).astype(complex)
    d, pairs = m[name]
    u = np.eye(d, dtype=complex)
    for a, b in pairs:
        u[[a, b]] = u[[b, a]]
    return u


def _axes(psi, wires, n):
    """psi [B, 2^n] with each wire as an axis of its own: the view and the wires' axes."""
    shape, at, axes = [psi.shape[0]], 0, {}
    for w in sorted(wires):
        shape += [1 << (w - at), 2]
        axes[w] = len(shape) - 1
        at = w + 1
    return psi.reshape(shape + [1 << (n - at)]), [axes[w] for w in wires]


def _apply(psi, m, wires, n):
    """m [d, d] or [B, d, d] on `wires` (wires[0] the most significant matrix bit) of psi [B, 2^n]."""
    if len(wires) == 1:
        v, _ = _axes(psi, wires, n)
        m = m.reshape(-1, 2, 2, 1, 1)
        a, b = v[:, :, 0], v[:, :, 1]
        return torch.stack([m[:, 0, 0] * a + m[:, 0, 1] * b, m[:, 1, 0] * a + m[:, 1, 1] * b], 2).reshape(psi.shape)
    v, ax = _axes(psi, wires, n)
    k = len(wires)
    v = v.movedim(ax, list(range(1, k + 1)))
    shape = v.shape
    v = torch.matmul(m, v.reshape(shape[0], 1 << k, -1)).reshape(shape).movedim(list(range(1, k + 1)), ax)
    return v.reshape(psi.shape)


def _cnot(psi, wires, n):
    v, (c, t) = _axes(psi, wires, n)
    v = v.clone()
    half = v.select(c, 1)
    half.copy_(half.flip(t - 1 if t > c else t))
    return v.reshape(psi.shape)


def _step(psi, op, angles, mats, n, inverse=False):
    name, wires, p, m = op
    if m is not None:
        return _apply(psi, torch.as_tensor(mats[m].astype(np.complex128), device=psi.device), wires, n)
    if name == "CNOT":
        return _cnot(psi, wires, n)
    if name in ("CZ", "SWAP", "Toffoli"):
        return _apply(psi, torch.as_tensor(_const(name), device=psi.device), wires, n)
    t = torch.zeros(1, dtype=torch.float64, device=psi.device) if p is None else angles[:, p]
    return _apply(psi, _mat(name, -t if inverse and p is not None else t), wires, n)


def _pauli(psi, word, wires, n):
    """P psi for psi [B, 2^n]."""
    for ch, w in zip(word, wires):
        v, _ = _axes(psi, [w], n)
        if ch == "X":
            v = v.flip(2)
        elif ch == "Y":
            v = torch.stack([-1j * v[:, :, 1], 1j * v[:, :, 0]], 2)
        elif ch == "Z":
            v = torch.stack([v[:, :, 0], -v[:, :, 1]], 2)
        psi = v.reshape(psi.shape)
    return psi


GEN = {"RX": "X", "RY": "Y", "RZ": "Z"}


def _reverse(lam, bras, ops, angles, n, groups):
    """Gradients [bras, params]: d<O>/dt = Im<bra|G|lam> for exp(-i t G / 2).  lam [B, N], bras [B * groups, N]
    (groups bras for each state, side by side)."""
    grad = torch.zeros(bras.shape[0], angles.shape[1], dtype=torch.float64, device=lam.device)
    both = torch.cat([lam, bras])
    rep = torch.cat([angles, angles.repeat_interleave(groups, 0)])
    B = lam.shape[0]
    for op in reversed(ops):
        name, wires, p, _ = op
        if p is not None:
            g = _pauli(both[:B], GEN[name], wires, n).repeat_interleave(groups, 0) if groups > 1 \
                else _pauli(both[:B], GEN[name], wires, n)
            grad[:, p] = torch.linalg.vecdot(both[B:], g).imag
        both = _step(both, op, rep, None, n, inverse=True)
    return grad


def _zero(B, n):
    psi = torch.zeros(B, 1 << n, dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1
    return psi


def _popcount_odd(x):
    for s in (32, 16, 8, 4, 2, 1):
        x = x ^ (x >> s)
    return (x & 1).bool()


def exact(case, seed):
    v, kind = _values(case, seed), case["kind"]
    if kind in ("execute", "gradient"):
        n = case["n"]
        angles = torch.tensor(v["angles"], device="cuda")[None]
        psi = _zero(1, n)
        for op in v["ops"]:
            psi = _step(psi, op, angles, None, n)
        if kind == "execute":
            words = [("ZZ", [q, (q + 1) % n]) for q in range(n)] + [("X", [q]) for q in range(n)]
            e = sum(c * torch.linalg.vecdot(psi, _pauli(psi, w, ws, n)).real.item() for c, (w, ws) in zip(v["coeffs"], words))
            return [np.float64(e), psi.abs().square()[0].cpu().numpy()]
        bras = torch.cat([_pauli(psi, "Z", [q], n) for q in range(case["nobs"])])
        return _reverse(psi, bras, v["ops"], angles, n, case["nobs"]).cpu().numpy()
    if kind == "batch":
        return _exact_batch(case, v)
    n = case["n"]
    psi = torch.view_as_complex(_state(case, seed).double())[None]
    if kind in ("circuit", "gates", "matrix"):
        angles = torch.tensor(v["angles"], device="cuda")[None]
        for op in v["ops"]:
            psi = _step(psi, op, angles, v["mats"], n)
        return torch.view_as_real(psi[0])
    if kind == "sample":
        p = psi[0].abs().square()
        wires = list(range(1, min(11, n), 2))
        t, ax = _axes(p[None], wires, n)
        keep = t.movedim(ax, list(range(len(wires)))).reshape(1 << len(wires), -1).sum(1)
        return [p, keep.cpu().numpy(), None]
    out, idx = [], torch.arange(1 << n, device="cuda")
    for word, wires in _words(case):
        x = z = ny = 0
        for ch, w in zip(word, wires):
            bit = 1 << (n - 1 - w)
            x |= bit if ch in "XY" else 0
            z |= bit if ch in "ZY" else 0
            ny += ch == "Y"
        r = torch.view_as_real(psi[0][idx ^ x].conj() * psi[0])
        r = (r[:, 0], -r[:, 1], -r[:, 0], r[:, 1])[ny & 3]
        out.append(torch.where(_popcount_odd(idx & z), -r, r).sum().item())
    out = np.array(out)
    return [out, np.float64((out * v["coeffs"]).sum())]


def _exact_batch(case, v):
    """Circuits of one shape share their structure and go through together, a few GB at a time."""
    circuit, shapes = case["circuit"], v["shapes"]
    per = 3 if circuit == "rot" else 2
    pat = np.cumsum([0] + [per * n * d for n, d in shapes])
    nob = [n if circuit == "rot" else 1 for n, _ in shapes]
    oat = np.cumsum([0] + nob)
    out = np.zeros(oat[-1])
    grad = np.zeros(pat[-1])
    for shape in sorted(set(shapes)):
        n, d = shape
        ops, np_ = _batch_ops(circuit, n, d)
        members = [c for c, s in enumerate(shapes) if s == shape]
        most = max(1, (1 << 24) >> n)
        for at in range(0, len(members), most):
            part = members[at:at + most]
            angles = torch.tensor(np.stack([v["angles"][pat[c]:pat[c + 1]] for c in part]), device="cuda")
            psi = _zero(len(part), n)
            for op in ops:
                psi = _step(psi, op, angles, None, n)
            bra = torch.zeros_like(psi)
            obs = [_batch_obs(circuit, n, v["coeffs"][c]) for c in part]
            for o in range(nob[part[0]]):
                w = torch.tensor([v["weights"][oat[c] + o] for c in part], device="cuda")
                val = torch.zeros(len(part), dtype=torch.float64, device="cuda")
                for t, (_, word, wires) in enumerate(obs[0][o]):
                    co = torch.tensor([obs[i][o][t][0] for i in range(len(part))], dtype=torch.float64, device="cuda")
                    term = _pauli(psi, word, wires, n)
                    val += co * torch.linalg.vecdot(psi, term).real
                    bra += (w * co)[:, None] * term
                out[[oat[c] + o for c in part]] = val.cpu().numpy()
            if case["grad"]:
                g = _reverse(psi, bra, ops, angles, n, 1).cpu().numpy()
                for i, c in enumerate(part):
                    grad[pat[c]:pat[c + 1]] = g[i]
    return [out, grad] if case["grad"] else out
