"""Fused passes by the length of their op lists: short lists run as a program
(a kernel parameter of at most 192 ops and 8 KiB of matrices), longer ones from
global memory.  Forward passes against numpy, the backward pass over two
uncompressed states against a numpy adjoint, at registers of several tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNIT = {"complex128": 2.0 ** -53, "complex64": 2.0 ** -24}


def apply(v, n, qubits, m):
    """v with m (matrix bit i on qubits[i]) applied, a copy."""
    k = len(qubits)
    axes = [n - 1 - q for q in reversed(qubits)]
    t = np.tensordot(np.asarray(m).reshape((2,) * (2 * k)), v.reshape((2,) * n), axes=(list(range(k, 2 * k)), axes))
    return np.moveaxis(t, list(range(k)), axes).reshape(-1)


def apply_gate(v, n, g, dagger=False):
    t, c, cv = g.get_target_index_list(), g.get_control_index_list(), g.get_control_value_list()
    m = g.get_matrix()
    for q, value in zip(c, cv):
        d = len(m)
        wide = np.eye(2 * d, dtype=np.complex128)
        wide[value * d:(value + 1) * d, value * d:(value + 1) * d] = m
        t, m = t + [q], wide
    return apply(v, n, t, m.conj().T if dagger else m)


def zero(n):
    v = np.zeros(1 << n, dtype=np.complex128)
    v[0] = 1.0
    return v


def unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def pairs_circuit(n, inside, count, seed):
    """Dense gates on pairs of the lowest `inside` qubits, every fourth gate a
    diagonal one that reaches outside (a matrix chosen by the tile)."""
    import qulacs
    from qulacs import gate as G
    rng = np.random.default_rng(seed)
    c = qulacs.QuantumCircuit(n)
    for q in range(n):
        c.add_H_gate(q)
    for k in range(count):
        if k % 4 == 3:
            a, b = int(rng.integers(inside)), int(rng.integers(inside, n))
            c.add_gate(G.DenseMatrix([a, b], np.diag(np.exp(1j * rng.uniform(0, 6, 4)))))
        else:
            a, b = (int(x) for x in rng.choice(inside, 2, replace=False))
            c.add_gate(G.DenseMatrix([a, b], unitary(rng, 4)))
    return c


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("count", [24, 56, 120, 320])
@pytest.mark.parametrize("compressed", [False, True])
def test_forward_passes_match_numpy(dtype, count, compressed):
    import qulacs
    from qulacs import _native
    n = 15
    c = pairs_circuit(n, 12, count, count)
    ref = zero(n)
    for g in c._gates:
        ref = apply_gate(ref, n, g)
    if compressed:
        st = qulacs.CompressedQuantumState(n, 13, dtype=dtype, eps_rel=1e-3, eps_abs=1e-7, flags=_native.QS_FLAG_QUIET)
        st.partition_and_register_circuit(c, 2, 0)
        st.apply_circuit()
        # one quantisation a pass, eps_rel |x| / 2 + eps_abs / 2 per component
        tol = (0.5e-3 + 0.5e-7 * 2 ** ((n + 1) / 2)) * st.get_stats()["passes"]
    else:
        st = qulacs.QuantumState(n, dtype=dtype)
        c.update_quantum_state(st)
        # four products an amplitude, each a few roundings, in every gate
        tol = 12 * UNIT[dtype] * len(c._gates)
    assert np.linalg.norm(st.get_vector() - ref) <= tol


def ansatz(n, layers, seed):
    """Rotations about every axis, some by exactly 0; ZZ, XX and YZ rotations
    of qubits far apart; CNOTs and a controlled gate across the register."""
    import qulacs
    from qulacs import gate as G
    rng = np.random.default_rng(seed)
    c = qulacs.ParametricQuantumCircuit(n)
    for q in range(n):
        c.add_H_gate(q)
    for layer in range(layers):
        for q in range(n):
            angle = 0.0 if rng.integers(6) == 0 else float(rng.uniform(0, 6))
            getattr(c, ("add_parametric_RX_gate", "add_parametric_RY_gate",
                        "add_parametric_RZ_gate")[int(rng.integers(3))])(q, angle)
        for a in range(n // 2):
            b = n - 1 - a
            ids = ([3, 3], [1, 1], [2, 3], [3, 3])[(a + layer) % 4]
            c.add_parametric_multi_Pauli_rotation_gate([a, b], ids, float(rng.uniform(0, 6)))
        for q in range(n - 1):
            c.add_CNOT_gate(q, q + 1)
        g = G.DenseMatrix(layer % n, unitary(rng, 2))
        g.add_control_qubit((layer + n // 2) % n, layer % 2)
        c.add_gate(g)
    return c


PAULI = {1: np.array([[0, 1], [1, 0]]), 2: np.array([[0, -1j], [1j, 0]]), 3: np.diag([1, -1])}


def generator(g):
    if hasattr(g, "axis"):
        return g.get_target_index_list(), PAULI["XYZ".index(g.axis) + 1]
    m = np.eye(1)
    for p in g._pids:
        m = np.kron(PAULI[p], m)
    return g.get_target_index_list(), m


def numpy_gradient(c, n, terms):
    """Energy and gradient of sum of coefficient * Z Z or X terms, backwards
    over psi and lambda = H psi: dE/dtheta = -Im <lambda| P |psi>."""
    psi = zero(n)
    for g in c._gates:
        psi = apply_gate(psi, n, g)
    lam = np.zeros_like(psi)
    for coef, p, qs in terms:
        t = psi
        for q in qs:
            t = apply(t, n, [q], PAULI[p])
        lam = lam + coef * t
    energy = np.vdot(psi, lam).real
    grad = []
    for k in reversed(range(len(c._gates))):
        g = c._gates[k]
        if k in c._param_pos:
            grad.append(-np.vdot(lam, apply(psi, n, *generator(g))).imag)
        psi, lam = apply_gate(psi, n, g, dagger=True), apply_gate(lam, n, g, dagger=True)
    return energy, np.array(grad[::-1])


@pytest.mark.parametrize("dtype,n", [("complex128", 12), ("complex128", 14), ("complex64", 13), ("complex64", 15)])
@pytest.mark.parametrize("layers", [1, 3, 9])
def test_backward_passes_match_numpy(monkeypatch, dtype, n, layers):
    """One layer fits a program; nine have more than 128 parameters and lists
    longer than a program.  The op-by-op path agrees as closely."""
    import qulacs
    from qulacs.torch import energy_and_gradient
    c = ansatz(n, layers, 10 * n + layers)
    terms = [(1.0, 3, (q, q + 1)) for q in range(n - 1)] + [(0.5, 1, (q,)) for q in range(n)]
    obs = qulacs.Observable(n)
    for coef, p, qs in terms:
        obs.add_operator(coef, " ".join(f"{'XYZ'[p - 1]} {q}" for q in qs))
    assert layers < 9 or c.get_parameter_count() > 128
    energy, grad = numpy_gradient(c, n, terms)
    # at most 12 roundings a gate and state (four products an amplitude), over
    # both states forwards and backwards, independent of one another
    tol = 12 * UNIT[dtype] * np.sqrt(4 * len(c._gates)) * sum(t[0] for t in terms)
    for sweeps in ("1", "0"):
        monkeypatch.setenv("QOMPSIM_DUAL_SWEEPS", sweeps)
        e, g = energy_and_gradient(c, obs, dtype)
        assert abs(e - energy) <= tol
        assert np.max(np.abs(np.asarray(g) - grad)) <= tol, sweeps
