"""Workloads of the state-vector engine for timing and comparing its outputs.

Every case goes through the package's public entry points:

* kind "apply"    -- a circuit on a CompressedQuantumState: reset to |0...0>,
                     apply_circuit, read the amplitudes into device memory
* kind "update"   -- a circuit on an uncompressed QuantumState
                     (QuantumCircuit.update_quantum_state, which plans on every
                     call), the state read through its device pointer
* kind "gradient" -- energy and gradient of a parametric circuit
                     (qulacs.torch.energy_and_gradient: forward, lambda = H psi,
                     backward over both states)
* kind "blocks"   -- a circuit fused to gates of up to four qubits
                     (QuantumCircuitOptimizer.optimize(block_size=4)) on a
                     CompressedQuantumState (apply_gates)
* kind "measure"  -- Pauli term values and block-wise samples of a compressed
                     state loaded from a vector

The circuits are the engine's workload families (GHZ fan-out, QFT of a basis
state, brickwork of random SU(2) and CZ, hardware-efficient ansatz, QAOA
MaxCut on a 3-regular graph), written here as plain gate lists so that
exact() can run the same lists in torch at 64 bits.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "compression-based-state-vector-simulator_b200"))

import qulacs  # noqa: E402
from qulacs import _native, gate as G  # noqa: E402
from qulacs.circuit import QuantumCircuitOptimizer  # noqa: E402


# ---------------------------------------------------------------- cases
def listed():
    return [
        # a short call: 256 blocks of which three are ever stored, so launches
        # and host work are what a caller waits for
        dict(name="ghz20", kind="apply", family="ghz", n=20, layers=1, block=12, inner=4, dtype="complex128"),
        # an ordinary QFT, the size of the tests and profiles
        dict(name="qft26", kind="apply", family="qft", n=26, layers=1, block=20, inner=4, dtype="complex128"),
        # the headline workload
        dict(name="qft30", kind="apply", family="qft", n=30, layers=1, block=20, inner=4, dtype="complex128"),
        # the same in single precision, an odd register and inner size
        dict(name="qft29_c64", kind="apply", family="qft", n=29, layers=1, block=20, inner=3, dtype="complex64"),
        # dense random states: every amplitude is mixed by every layer
        dict(name="brickwork26_c64", kind="apply", family="brickwork", n=26, layers=14, block=18, inner=4,
             dtype="complex64"),
        dict(name="brickwork25", kind="apply", family="brickwork", n=25, layers=8, block=17, inner=3,
             dtype="complex128"),
        # a variational optimiser's energy state: diagonal layers between mixers
        dict(name="qaoa26_c64", kind="apply", family="qaoa", n=26, layers=3, block=20, inner=4, dtype="complex64"),
        # the uncompressed state, as a reference run or a training loop uses it
        dict(name="update_qft27", kind="update", family="qft", n=27, layers=1, dtype="complex128"),
        dict(name="update_brickwork27_c64", kind="update", family="brickwork", n=27, layers=6, dtype="complex64"),
        # one step of a variational training loop: forward and backward
        dict(name="gradient21", kind="gradient", family="hea", n=21, layers=4, dtype="complex128"),
        # circuits fused to four-qubit gates (tensor cores)
        dict(name="blocks24_c64", kind="blocks", family="brickwork", n=24, layers=4, block=16, inner=4,
             dtype="complex64"),
        # reading results off a compressed state
        dict(name="measure23", kind="measure", family="random", n=23, layers=1, block=15, inner=4,
             dtype="complex128", shots=20000),
    ]


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "apply", "update", "update", "gradient", "blocks", "measure"])
    dtype = rng.choice(["complex128", "complex64"])
    if kind == "apply":
        family = rng.choice(["ghz", "qft", "qft", "brickwork", "brickwork", "qaoa"])
        n, layers = {
            "ghz": (rng.randint(16, 20), 1),
            "qft": (rng.randint(18, 29), 1),
            "brickwork": (rng.randint(19, 26), rng.randint(3, 14)),
            "qaoa": (2 * rng.randint(9, 13), rng.randint(1, 4)),
        }[family]
        return dict(kind=kind, family=family, n=n, layers=layers, block=n - rng.randint(5, 9),
                    inner=rng.randint(2, 5), dtype=dtype)
    if kind == "update":
        family = rng.choice(["qft", "brickwork", "hea"])
        return dict(kind=kind, family=family, n=rng.randint(17, 27),
                    layers=1 if family == "qft" else rng.randint(2, 8), dtype=dtype)
    if kind == "gradient":
        return dict(kind=kind, family="hea", n=rng.randint(14, 22), layers=rng.randint(2, 5), dtype="complex128")
    n = rng.randint(18, 23)
    if kind == "blocks":
        return dict(kind=kind, family="brickwork", n=n, layers=rng.randint(2, 5), block=n - rng.randint(5, 8),
                    inner=rng.randint(3, 5), dtype=dtype)
    return dict(kind=kind, family="random", n=n, layers=1, block=n - rng.randint(5, 8), inner=4, dtype=dtype,
                shots=rng.randint(1000, 50000))


# ---------------------------------------------------------------- gate lists
def haar_su2(rng):
    z = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
    q, r = np.linalg.qr(z)
    q = q * (np.diag(r) / np.abs(np.diag(r)))
    return q / np.sqrt(np.linalg.det(q))


def basis_input(n, rng):
    return int(rng.integers(1, 1 << n))


def gate_list(case, seed):
    """The circuit as plain tuples: ("X", q), ("H", q), ("U", q, 2x2 matrix),
    ("RX" / "RY" / "RZ", q, angle), ("CP", control, target, angle),
    ("CX" / "CZ" / "SWAP", a, b), ("RZZ", a, b, angle)."""
    rng = np.random.default_rng(seed)
    n, layers = case["n"], case["layers"]
    g = []
    if case["family"] in ("ghz", "qft"):
        x = basis_input(n, rng)
        g += [("X", q) for q in range(n) if (x >> q) & 1]
    if case["family"] == "ghz":
        g.append(("H", 0))
        g += [("CX", 0, q) for q in range(1, n)]
    elif case["family"] == "qft":
        for j in reversed(range(n)):
            g.append(("H", j))
            g += [("CP", j, k, 2.0 * math.pi / 2 ** (j - k + 1)) for k in reversed(range(j))]
        g += [("SWAP", i, n - 1 - i) for i in range(n // 2)]
    elif case["family"] == "brickwork":
        for layer in range(layers):
            g += [("U", q, haar_su2(rng)) for q in range(n)]
            g += [("CZ", a, a + 1) for a in range(layer % 2, n - 1, 2)]
    elif case["family"] == "hea":
        for _ in range(layers):
            for q in range(n):
                g.append(("RY", q, float(rng.uniform(0.0, 2.0 * math.pi))))
                g.append(("RZ", q, float(rng.uniform(0.0, 2.0 * math.pi))))
            g += [("CX", q, q + 1) for q in range(n - 1)]
    elif case["family"] == "qaoa":
        p = [int(v) for v in rng.permutation(n)]
        edges = [(p[i], p[(i + 1) % n]) for i in range(n)] + [(p[i], p[i + n // 2]) for i in range(n // 2)]
        g += [("H", q) for q in range(n)]
        for _ in range(layers):
            gamma, beta = rng.uniform(0.0, math.pi, size=2)
            g += [("RZZ", min(e), max(e), float(gamma)) for e in edges]
            g += [("RX", q, float(beta)) for q in range(n)]
    return g


def circuit_of(case, gates, parametric=False):
    c = qulacs.ParametricQuantumCircuit(case["n"]) if parametric else qulacs.QuantumCircuit(case["n"])
    for g in gates:
        op, a = g[0], g[1]
        if op == "X":
            c.add_X_gate(a)
        elif op == "H":
            c.add_H_gate(a)
        elif op == "U":
            c.add_gate(G.DenseMatrix(a, g[2]))
        elif op == "RX":
            c.add_RX_gate(a, g[2])
        elif op in ("RY", "RZ"):
            add = {("RY", False): "add_RY_gate", ("RZ", False): "add_RZ_gate",
                   ("RY", True): "add_parametric_RY_gate", ("RZ", True): "add_parametric_RZ_gate"}[op, parametric]
            getattr(c, add)(a, g[2])
        elif op == "CP":
            d = G.DenseMatrix(g[2], np.diag([1.0, np.exp(1j * g[3])]))
            d.add_control_qubit(a, 1)
            c.add_gate(d)
        elif op == "RZZ":
            ph = np.exp(0.5j * g[3])
            c.add_gate(G.DenseMatrix([a, g[2]], np.diag([ph, np.conj(ph), np.conj(ph), ph])))
        else:
            {"CX": c.add_CNOT_gate, "CZ": c.add_CZ_gate, "SWAP": c.add_SWAP_gate}[op](a, g[2])
    return c


def observable_terms(n):
    """sum_i Z_i Z_{i+1} + 0.5 sum_i X_i, as (coefficient, Pauli, qubits)."""
    return [(1.0, "Z", (i, i + 1)) for i in range(n - 1)] + [(0.5, "X", (i,)) for i in range(n)]


def observable_of(n):
    obs = qulacs.Observable(n)
    for coef, p, qs in observable_terms(n):
        obs.add_operator(coef, " ".join(f"{p} {q}" for q in qs))
    return obs


def random_vector(n, seed):
    """A normalised vector with the spread of a random circuit's amplitudes."""
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(2 << n).view(np.complex128)
    return v / np.linalg.norm(v)


# ---------------------------------------------------------------- one pass
class DeviceArray:
    """The device memory of an uncompressed state, for torch."""

    def __init__(self, state, n, dtype):
        self.state = state
        self.__cuda_array_interface__ = {"shape": (1 << n,), "typestr": "<c16" if dtype == "complex128" else "<c8",
                                         "data": (state.device_pointer(), False), "version": 3, "strides": None}


def compressed_state(case):
    return qulacs.CompressedQuantumState(case["n"], case["block"], dtype=case["dtype"], eps_rel=1e-3, eps_abs=1e-7,
                                         flags=_native.QS_FLAG_QUIET)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"case": case, "seed": seed}
    if kind == "measure":
        s["observable"] = observable_of(n)
        s["state"] = compressed_state(case)
        s["state"].load(random_vector(n, seed))
        return s
    gates = gate_list(case, seed)
    if kind == "gradient":
        s["circuit"] = circuit_of(case, gates, parametric=True)
        s["observable"] = observable_of(n)
        return s
    circuit = circuit_of(case, gates)
    if kind == "update":
        QuantumCircuitOptimizer().optimize(circuit, block_size=2)
        s["circuit"] = circuit
        s["state"] = qulacs.QuantumState(n, dtype=case["dtype"])
        s["vector"] = torch.as_tensor(DeviceArray(s["state"], n, case["dtype"]), device="cuda")
        return s
    QuantumCircuitOptimizer(sv_block_size=case["block"]).optimize(circuit, block_size=4 if kind == "blocks" else 2)
    s["state"] = compressed_state(case)
    if kind == "blocks":
        s["gates"] = circuit.get_gate_list()
    else:
        s["state"].partition_and_register_circuit(circuit, case["inner"], 0)
    s["amplitudes"] = torch.empty(1 << n, dtype=torch.complex128, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind, n = case["kind"], case["n"]
    if kind == "gradient":
        from qulacs.torch import energy_and_gradient
        energy, grad = energy_and_gradient(s["circuit"], s["observable"], case["dtype"])
        return {"energy": energy, "gradient": grad}
    state = s["state"]
    if kind == "measure":
        return {"terms": s["observable"].get_term_values(state),
                "samples": np.asarray(state.sampling_blockwise(case["shots"], s["seed"] & 0xFFFF), dtype=np.int64)}
    state.set_zero_state()
    if kind == "update":
        s["circuit"].update_quantum_state(state)
        return {"vector": s["vector"]}
    if kind == "blocks":
        state.apply_gates(s["gates"], case["inner"])
    else:
        state.apply_circuit()
    state.get_amplitudes_to(s["amplitudes"].data_ptr(), 0, 1 << n)
    return {"amplitudes": s["amplitudes"]}


def work(case):
    """Bytes: the result written once (and, where a state is the input, read
    once).  Flops: the gates' arithmetic on the amplitudes that they change."""
    n, dim = case["n"], float(1 << case["n"])
    amp = 16.0 if case["dtype"] == "complex128" else 8.0
    if case["kind"] == "measure":
        terms = len(observable_terms(n))
        return {"bytes": amp * dim + 8.0 * case["shots"], "flops": (8.0 * terms + 4.0) * dim}
    per = {"X": 0.0, "H": 4.0, "U": 14.0, "RX": 8.0, "RY": 6.0, "RZ": 6.0, "CP": 1.5, "CX": 0.0, "CZ": 0.5,
           "SWAP": 0.0, "RZZ": 6.0}
    flops = sum(per[g[0]] for g in gate_list(case, 0)) * dim
    if case["kind"] == "gradient":
        terms = len(observable_terms(n))
        params = 2 * n * case["layers"]
        return {"bytes": 4 * amp * dim, "flops": 3.0 * flops + (12.0 * terms + 8.0 * params) * dim}
    # compressed states are read out as complex128 amplitudes
    return {"bytes": (amp if case["kind"] == "update" else 16.0) * dim, "flops": flops}


# ---------------------------------------------------------------- 64-bit values
def matrix_of(g):
    """2x2 matrix of a one-qubit gate (Qulacs sign convention: exp(+i angle P / 2))."""
    op = g[0]
    if op == "X":
        return np.array([[0, 1], [1, 0]], dtype=np.complex128)
    if op == "H":
        return np.array([[1, 1], [1, -1]], dtype=np.complex128) / math.sqrt(2.0)
    if op == "U":
        return np.asarray(g[2])
    c, s = math.cos(g[2] / 2), math.sin(g[2] / 2)
    if op == "RX":
        return np.array([[c, 1j * s], [1j * s, c]])
    if op == "RY":
        return np.array([[c, s], [-s, c]], dtype=np.complex128)
    return np.diag([c + 1j * s, c - 1j * s])


def bits(v, n, qubits):
    """v viewed with one axis of length 2 per listed qubit (ascending), and
    the axes, as {qubit: axis}."""
    shape, axis, top = [], {}, n
    for q in sorted(qubits, reverse=True):
        shape += [1 << (top - q - 1), 2]
        axis[q] = len(shape) - 1
        top = q
    shape.append(1 << top)
    return v.view(shape), axis


def part(w, axis, values):
    """The part of w where each listed qubit has the given value."""
    index = [slice(None)] * w.dim()
    for q, b in values.items():
        index[axis[q]] = b
    return w[tuple(index)]


def apply_exact(v, n, g):
    op = g[0]
    if op in ("CP", "CX", "CZ", "SWAP", "RZZ"):
        a, b = g[1], g[2]
        w, ax = bits(v, n, (a, b))
        if op == "CP":
            part(w, ax, {a: 1, b: 1}).mul_(complex(np.exp(1j * g[3])))
        elif op == "CZ":
            part(w, ax, {a: 1, b: 1}).neg_()
        elif op == "RZZ":
            ph = complex(np.exp(0.5j * g[3]))
            for x in (0, 1):
                for y in (0, 1):
                    part(w, ax, {a: x, b: y}).mul_(ph if x == y else ph.conjugate())
        else:
            p, q = ({a: 1, b: 0}, {a: 1, b: 1}) if op == "CX" else ({a: 1, b: 0}, {a: 0, b: 1})
            t = part(w, ax, p).clone()
            part(w, ax, p).copy_(part(w, ax, q))
            part(w, ax, q).copy_(t)
        return
    m = matrix_of(g)
    w, ax = bits(v, n, (g[1],))
    x, y = part(w, ax, {g[1]: 0}), part(w, ax, {g[1]: 1})
    t = x * complex(m[0, 0])
    t.add_(y, alpha=complex(m[0, 1]))
    y.mul_(complex(m[1, 1])).add_(x, alpha=complex(m[1, 0]))
    x.copy_(t)


def inverse_of(g):
    if g[0] in ("RX", "RY", "RZ"):
        return (g[0], g[1], -g[2])
    return g


def apply_pauli(v, n, p, qs):
    """The Pauli string (one letter on each listed qubit) applied to v."""
    out = v.clone()
    for q in qs:
        w, ax = bits(out, n, (q,))
        if p == "Z":
            part(w, ax, {q: 1}).neg_()
        elif p == "X":
            apply_exact(out, n, ("X", q))
        else:
            apply_exact(out, n, ("U", q, np.array([[0, -1j], [1j, 0]])))
    return out


def zero_vector(n, device):
    v = torch.zeros(1 << n, dtype=torch.complex128, device=device)
    v[0] = 1.0
    return v


def exact_gradient(case, gates, device):
    n = case["n"]
    psi = zero_vector(n, device)
    for g in gates:
        apply_exact(psi, n, g)
    lam = torch.zeros_like(psi)
    for coef, p, qs in observable_terms(n):
        lam.add_(apply_pauli(psi, n, p, qs), alpha=coef)
    energy = float(torch.vdot(psi, lam).real)
    grad = []
    for g in reversed(gates):
        if g[0] in ("RX", "RY", "RZ"):
            grad.append(-float(torch.vdot(lam, apply_pauli(psi, n, g[0][1], (g[1],))).imag))
        inv = inverse_of(g)
        apply_exact(psi, n, inv)
        apply_exact(lam, n, inv)
    return {"energy": energy, "gradient": np.array(grad[::-1])}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    n = case["n"]
    if case["kind"] == "measure":
        v = torch.from_numpy(random_vector(n, seed)).to(device)
        norm = float(torch.vdot(v, v).real)
        terms = [complex(torch.vdot(v, apply_pauli(v, n, p, qs))) / norm for _, p, qs in observable_terms(n)]
        return {"terms": np.array(terms), "samples": None}
    if case["family"] == "qft":
        # amplitude k of the transform of |x>: 2^(-n/2) e^(2 pi i x k / 2^n)
        x = basis_input(n, np.random.default_rng(seed))
        v = torch.empty(1 << n, dtype=torch.complex128, device=device)
        for first in range(0, 1 << n, 1 << 24):
            k = torch.arange(first, min(first + (1 << 24), 1 << n), device=device, dtype=torch.int64)
            angle = ((x * k) & ((1 << n) - 1)).double() * (2.0 * math.pi / (1 << n))
            v[first:first + k.numel()] = torch.polar(torch.full_like(angle, 2.0 ** (-n / 2)), angle)
    else:
        gates = gate_list(case, seed)
        if case["kind"] == "gradient":
            return exact_gradient(case, gates, device)
        v = zero_vector(n, device)
        for g in gates:
            apply_exact(v, n, g)
    return {"vector": v} if case["kind"] == "update" else {"amplitudes": v}
