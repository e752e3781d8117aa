"""The oracle that stands in where the reference's csim kernels are not built
(oracle/dense_oracle.cpp), against the golden states that csim wrote, full
matrix products and csim itself where it is there (CPU only)."""
import numpy as np
import pytest

import helpers
from oracle import csim_ref


@pytest.fixture()
def dense(monkeypatch):
    monkeypatch.setattr(csim_ref, "_lib", csim_ref.dense_kernels())


@pytest.mark.parametrize("key", sorted(helpers.golden_circuits()))
def test_golden_states(dense, key):
    c = helpers.build_circuit(key)
    v = csim_ref.run_circuit(c.get_qubit_count(), c._gates)
    assert np.abs(v - helpers.golden_states()[key]).max() < 1e-13
    assert abs(csim_ref.norm_squared(v) - 1.0) < 1e-12
    assert abs(csim_ref.inner_product(v, v) - 1.0) < 1e-12


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_gate_form(dense, seed):
    """Controls of either value, two targets in either order, named gates."""
    import qulacs
    from qulacs import gate as G
    from qulacs._gates import full_matrix
    rng = np.random.default_rng(seed)
    n = 6
    gates = list(helpers.random_circuit(n, 40, seed=seed)._gates)
    for k in range(20):
        a, b, c, d = (int(q) for q in rng.permutation(n)[:4])
        g = G.DenseMatrix([a, b] if k % 2 else [a], rng.normal(size=(2 + 2 * (k % 2),) * 2))
        g.add_control_qubit(c, k % 3 % 2)
        if k % 4 == 0:
            g.add_control_qubit(d, 1)
        gates.append(g)
    for g in gates:
        v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
        got = csim_ref.apply_gates(v.copy(), [g])
        m, order = full_matrix(g)
        at = np.arange(1 << n)
        row = sum(((at >> q) & 1) << i for i, q in enumerate(order))
        rest = at & ~sum(1 << q for q in order)
        want = sum(m[row, r] * v[rest | sum(((r >> i) & 1) << q for i, q in enumerate(order))] for r in range(len(m)))
        assert np.abs(got - want).max() < 1e-12
