"""Tile-pass kernels at their edges: the payloads a pass writes against the C
statement of the codec at every chunk size, passes too long for a program
against the ones that fit, amplitudes read to device memory at any 8-byte
alignment, and Pauli sums on tiles smaller than a CTA."""
import struct

import numpy as np
import pytest

from oracle import codec

pytestmark = pytest.mark.gpu


def _dense(n, gates):
    from qulacs._gates import full_matrix
    v = np.zeros((2,) * n, dtype=np.complex128)
    v[(0,) * n] = 1.0
    for g in gates:
        m, order = full_matrix(g)
        k = len(order)
        axes = [n - 1 - q for q in reversed(order)]
        t = np.tensordot(m.reshape((2,) * (2 * k)), v, axes=(list(range(k, 2 * k)), axes))
        v = np.moveaxis(t, list(range(k)), axes)
    return v.reshape(-1)


def _state(n, B, dtype, eps_rel=1e-3, eps_abs=1e-7):
    import qulacs
    from qulacs import _native
    return qulacs.CompressedQuantumState(n, B, dtype=dtype, eps_rel=eps_rel, eps_abs=eps_abs,
                                         flags=_native.QS_FLAG_QUIET)


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("C", [4, 5, 6, 7, 8])
# eps_abs 1e-4 leaves small amplitudes in the linear region, 1e-12 puts all in
# the logarithmic one; eps_rel 2^-23 takes the paths without signed rounding
@pytest.mark.parametrize("eps_rel,eps_abs", [(1e-3, 1e-4), (1e-3, 1e-12), (2.0 ** -23, 1e-9)])
def test_pass_payloads_match_the_codec_statement(monkeypatch, C, dtype, eps_rel, eps_abs):
    from qompsim import circuits as Q
    monkeypatch.setenv("QOMPSIM_CHUNK_LOG2", str(C))
    n, B = 11, 8
    st = _state(n, B, dtype, eps_rel, eps_abs)
    st.partition_and_register_circuit(Q.brickwork(n, 3, seed=C), 3, 0)
    st.apply_circuit()
    assert st.get_stats()["chunk_log2"] == C
    blob = st.export_store()
    _, _, _, hC, f64, m, L, nb, nchunks, _ = struct.unpack_from("<8s4I2i3Q", blob)
    assert hC == C and nchunks == 1 << (n - C)
    off = struct.calcsize("<8s4I2i3Q")
    mask = np.frombuffer(blob, np.uint8, nb, off)
    off += nb + 8 * nb
    meta = np.frombuffer(blob, np.dtype([("offset", "<u8"), ("base", "<i4"), ("width", "<u4")]), nchunks, off)
    arena = off + 16 * nchunks
    values = st.get_amplitudes(0, 1 << n, renormalize=False).view(np.float64)
    per = 2 << C
    for k in range(nchunks):
        if not mask[k >> (B - C)]:
            continue
        got = values[k * per:(k + 1) * per].astype(np.float64 if f64 else np.float32)
        base, width = int(meta[k]["base"]), int(meta[k]["width"])
        nbytes = codec.payload_bytes(C, width)
        words = np.frombuffer(blob, np.uint32, nbytes // 4, arena + int(meta[k]["offset"])).copy()
        want = codec.decode_chunk(words, C, base, width, m, L, bool(f64))
        assert np.array_equal(got, want)
        # quantise(dequantise(c)) == c: encoding the values gives the chunk back
        again = codec.encode_chunk(got, C, m, L)
        assert (again[1], again[2]) == (base, width) and np.array_equal(np.asarray(again[0])[:nbytes // 4], words)


@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-11), ("complex64", 2e-4)])
@pytest.mark.parametrize("gates", [40, 900])
def test_long_op_lists_match_dense(dtype, tol, gates):
    """40 gates fit a program, 900 two-qubit gates on 13 qubits need more ops,
    sweeps and matrices than one holds.  Tolerance: `gates` products of
    rounding 2^-53 (2^-24) with a factor of 100 (5) to spare."""
    import qulacs
    from qulacs import gate as G
    rng = np.random.default_rng(gates)
    n = 13
    c = qulacs.QuantumCircuit(n)
    for _ in range(gates):
        a, b = (int(q) for q in rng.choice(n, 2, replace=False))
        u, _ = np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))
        c.add_gate(G.DenseMatrix([a, b], u))
    ref = _dense(n, c._gates)
    s = qulacs.QuantumState(n, dtype=dtype)
    c.update_quantum_state(s)
    assert np.linalg.norm(s.get_vector() - ref) < tol
    st = _state(n, 9, dtype, eps_rel=1e-6, eps_abs=1e-9)
    st.partition_and_register_circuit(c, 4, 0)
    st.apply_circuit()
    # a pass quantises once: eps_rel / 2 of the norm and eps_abs / 2 per component
    budget = (0.5e-6 + 0.5e-9 * 2 ** ((n + 1) / 2)) * st.get_stats()["passes"]
    assert np.linalg.norm(st.get_vector() - ref) < budget + tol


def test_readout_to_device_memory_alignment():
    import torch
    from qompsim import circuits as Q
    n = 12
    for dtype in ("complex128", "complex64"):
        st = _state(n, 9, dtype)
        st.partition_and_register_circuit(Q.brickwork(n, 2, seed=1), 3, 0)
        st.apply_circuit()
        want = st.get_amplitudes(0, 1 << n).view(np.float64)
        buf = torch.zeros((2 << n) + 2, dtype=torch.float64, device="cuda")
        for shift in (0, 1, 2):
            buf.fill_(-7.0)
            st.get_amplitudes_to(buf.data_ptr() + 8 * shift, 0, 1 << n)
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + (2 << n)], want)
            assert (got[:shift] == -7.0).all() and (got[shift + (2 << n):] == -7.0).all()
        # part of the state
        st.get_amplitudes_to(buf.data_ptr(), 256, 512)
        assert np.array_equal(buf[:1024].cpu().numpy(), want[512:1536])


@pytest.mark.parametrize("n,B", [(5, 4), (6, 5), (9, 6), (13, 9)])
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_pauli_sums_on_small_tiles(n, B, dtype):
    rng = np.random.default_rng(n)
    v = rng.normal(size=2 << n).view(np.complex128)
    v /= np.linalg.norm(v)
    st = _state(n, B, dtype)
    st.load(v)
    w = st.get_amplitudes(0, 1 << n, renormalize=False)
    x = np.arange(1 << n)
    xs = [0, 0, 1, 1 << (n - 1), 3, 0, 5]
    zs = [0, (1 << n) - 1, 0, 0, 1 << (n - 1), 2, 4]
    got = st._pauli_sums(xs, zs)
    for xm, zm, g in zip(xs, zs, got):
        sign = np.where([bin(int(i) & zm).count("1") & 1 for i in x], -1.0, 1.0)
        assert abs(g - np.sum(np.conj(w[x ^ xm]) * sign * w)) < 1e-12
