"""Passes that change the order of the qubits (plan_layout_passes): the planner
against direct gate application on the CPU, and on the GPU the reordered tail
against the fixed-order one and a dense FP64 vector."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "compression-based-state-vector-simulator_b200", "csrc")
CUDA = "/usr/local/cuda"


@pytest.mark.parametrize("seed", [1, 2])
def test_layout_plan_keeps_the_state(tmp_path, seed):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("no host C++ compiler or CUDA headers")
    exe = tmp_path / "layout_plan_check"
    cmd = [gxx, "-O1", "-std=c++17", "-w", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", str(exe),
           os.path.join(HERE, "layout_plan_check.cpp"), "-L", os.path.join(CUDA, "lib64"), "-lcudart",
           "-Wl,--unresolved-symbols=ignore-all", "-Wl,-rpath," + os.path.join(CUDA, "lib64")]
    env = dict(os.environ)
    env.pop("CXX", None)
    r = subprocess.run(cmd, capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe), str(seed), "150"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "layout ok" in r.stdout, r.stdout + r.stderr


def _dense(n, gates):
    """The gates applied one by one to |0...0> in numpy."""
    from qulacs._gates import full_matrix
    v = np.zeros((2,) * n, dtype=np.complex128)
    v[(0,) * n] = 1.0
    for g in gates:
        m, order = full_matrix(g)
        k = len(order)
        axes = [n - 1 - q for q in reversed(order)]   # matrix bit k-1 first
        t = np.tensordot(m.reshape((2,) * (2 * k)), v, axes=(list(range(k, 2 * k)), axes))
        v = np.moveaxis(t, list(range(k)), axes)
    return v.reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n,B,layers", [(14, 9, 8), (17, 11, 10), (19, 12, 12)])
def test_reordered_tail_matches_dense_and_fixed_order(monkeypatch, n, B, layers, dtype):
    """Brickwork (a chain: the reordering tail takes fewer passes): within the
    codec's error budget of a dense vector, same masks and stage count as the
    fixed order, and an error no larger than the fixed order's but for the
    scatter of 2^14 and more roundings (well under 5 % of their norm)."""
    import qulacs
    from qulacs import _native
    from qulacs.circuit import QuantumCircuitOptimizer
    from qompsim import circuits as C
    c = C.brickwork(n, layers, seed=n)
    QuantumCircuitOptimizer(sv_block_size=B).optimize(c, block_size=2)
    ref = _dense(n, c._gates)
    got = {}
    for env in ("0", "1"):
        monkeypatch.setenv("QOMPSIM_LAYOUT", env)
        st = qulacs.CompressedQuantumState(n, B, dtype=dtype, eps_rel=1e-3, eps_abs=1e-7, flags=_native.QS_FLAG_QUIET)
        st.partition_and_register_circuit(c, 4, 0)
        st.apply_circuit()
        err = np.linalg.norm(st.get_vector() - ref)
        got[env] = (err, st.get_zero_mask().tolist(), st.get_stats()["passes"], len(st.get_SV_bytes_history()))
    assert got["1"][2] <= got["0"][2]
    if n >= 17:
        assert got["1"][2] < got["0"][2]
    assert got["1"][1] == got["0"][1] and got["1"][3] == got["0"][3]
    # one quantisation a pass, each at most eps_rel |x| / 2 + eps_abs / 2 per
    # component: the relative errors of the passes add up at worst
    for env in ("0", "1"):
        assert got[env][0] <= (0.5e-3 + 0.5e-7 * 2 ** ((n + 1) / 2)) * got[env][2]
    assert got["1"][0] <= 1.05 * got["0"][0]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_arena_that_holds_the_fixed_order_is_enough(monkeypatch, dtype):
    """A chain whose amplitudes differ in size with the upper qubits only, so
    that chunks of the lower ones pack best: in arenas from too small to roomy,
    wherever the fixed order runs, so does the default, with the same masks."""
    import qulacs
    from qulacs import _native
    from qulacs.circuit import QuantumCircuitOptimizer
    n, B = 16, 10
    c = qulacs.QuantumCircuit(n)
    for q in range(n):
        c.add_H_gate(q) if q < 8 else c.add_RY_gate(q, 0.4)
    for layer in range(9):
        for q in range(n):
            c.add_RX_gate(q, 1e-3 * (1 + q / n))
        for a in range(layer % 2, n - 1, 2):
            c.add_CZ_gate(a, a + 1)
    QuantumCircuitOptimizer(sv_block_size=B).optimize(c, block_size=2)

    def run(layout, arena):
        monkeypatch.setenv("QOMPSIM_LAYOUT", layout)
        monkeypatch.setenv("QOMPSIM_ARENA_BYTES", str(arena))
        st = qulacs.CompressedQuantumState(n, B, dtype=dtype, eps_rel=1e-3, eps_abs=1e-7, flags=_native.QS_FLAG_QUIET)
        st.partition_and_register_circuit(c, 4, 0)
        try:
            st.apply_circuit()
        except _native.QompsimError as e:
            assert e.status == _native.QS_ERR_CAPACITY
            return None
        return st.get_zero_mask().tolist(), sum(st.get_block_bytes())

    final = run("0", 8 << n)[1]
    fits = []
    for percent in range(90, 131):
        arena = final * percent // 100
        fixed = run("0", arena)
        fits.append(fixed is not None)
        if fixed is not None:
            got = run("1", arena)
            assert got is not None and got[0] == fixed[0], percent
    assert fits[-1] and not fits[0]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_byte_totals_of_a_reordered_tail(monkeypatch, dtype):
    """Every stage has a total in both orders; the last is the state's, the
    same in both up to the codes that differ, and none passes the widest store
    of a normalised state (16 bits a component and a 16-byte header a chunk)."""
    import qulacs
    from qulacs import _native
    from qulacs.circuit import QuantumCircuitOptimizer
    from qompsim import circuits as C
    n, B = 17, 11
    c = C.brickwork(n, 10, seed=n)
    QuantumCircuitOptimizer(sv_block_size=B).optimize(c, block_size=2)
    last = {}
    for env in ("0", "1"):
        monkeypatch.setenv("QOMPSIM_LAYOUT", env)
        st = qulacs.CompressedQuantumState(n, B, dtype=dtype, eps_rel=1e-3, eps_abs=1e-7, flags=_native.QS_FLAG_QUIET)
        st.partition_and_register_circuit(c, 4, 0)
        st.apply_circuit()
        history = st.get_SV_bytes_history()
        assert len(history) == st.get_stats()["stages"] + 1
        assert history[-1] == sum(int(b) for b in st.get_block_bytes())
        assert st.get_max_SV_bytes() == max(history) <= (1 << (n - 8)) * (1024 + 16)
        last[env] = history[-1]
    # a chunk's width moves by a bit at most (its largest code by the passes'
    # relative error, far below a factor of two), so its payload by one row
    assert abs(last["1"] - last["0"]) <= (1 << (n - 8)) * 128
