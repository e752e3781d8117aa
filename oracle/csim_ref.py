"""ORACLE (test infrastructure only): the reference's FP64 csim kernels.

Loads oracle/_ref/libcsim_ref.so (built from the reference's src/csim by
oracle/Makefile) and applies a qulacs gate list to a dense complex128 vector
with the kernel the reference would call for that gate:

* "CNOT" / "CZ" / "SWAP"  -> CNOT_gate / CZ_gate / SWAP_gate
  (src/csim/update_ops_named_{CNOT,CZ,SWAP}.cpp)
* a matrix gate without controls -> single_qubit_dense_matrix_gate or
  double_qubit_dense_matrix_gate_c (gate_matrix.cpp:128-160 dispatch)
* with controls -> multi_qubit_control_multi_qubit_dense_matrix_gate

Where that library is not built (the reference is not mounted), the same calls
run this package's own plain statement of them (dense_oracle.cpp, in
oracle/build/liboracle.so); available() tells which one checks.
"""
from __future__ import annotations

import ctypes as ct
import os
from typing import Sequence

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "_ref", "libcsim_ref.so")

_lib = None


def available() -> bool:
    return os.path.exists(LIB_PATH)


class _Kernels:
    """The library's functions by their names without the prefix."""

    def __init__(self, library, prefix):
        P = ct.c_void_p
        U = ct.c_uint
        U64 = ct.c_uint64
        for name, restype, argtypes in (
                ("dense1", None, [U, P, P, U64]), ("dense2", None, [U, U, P, P, U64]),
                ("dense_multi", None, [P, U, P, P, U64]), ("controlled", None, [P, P, U, P, U, P, P, U64]),
                ("cnot", None, [U, U, P, U64]), ("cz", None, [U, U, P, U64]), ("swap", None, [U, U, P, U64]),
                ("norm_squared", ct.c_double, [P, U64]), ("inner_product", None, [P, P, U64, P]),
                ("init_zero", None, [P, U64]), ("max_threads", ct.c_int, [])):
            f = getattr(library, prefix + name)
            f.restype, f.argtypes = restype, argtypes
            setattr(self, name, f)


def dense_kernels() -> _Kernels:
    """dense_oracle.cpp's functions."""
    from . import codec
    return _Kernels(codec.lib(), "qsor_dense_")


def lib() -> _Kernels:
    global _lib
    if _lib is None:
        _lib = _Kernels(ct.CDLL(LIB_PATH), "csimref_") if available() else dense_kernels()
    return _lib


def zero_state(n: int) -> np.ndarray:
    s = np.empty(1 << n, dtype=np.complex128)
    lib().init_zero(s.ctypes.data, s.size)
    return s


def _ptr(a):
    return a.ctypes.data


def apply_gate(state: np.ndarray, g) -> None:
    assert state.dtype == np.complex128 and state.flags.c_contiguous
    L = lib()
    dim = state.size
    name = g.get_name()
    t = g.get_target_index_list()
    c = g.get_control_index_list()
    cv = g.get_control_value_list()
    if name == "CNOT":
        L.cnot(c[0], t[0], _ptr(state), dim)
        return
    if name == "CZ":
        L.cz(c[0], t[0], _ptr(state), dim)
        return
    if name == "SWAP":
        L.swap(t[0], t[1], _ptr(state), dim)
        return
    m = np.ascontiguousarray(g.get_matrix(), dtype=np.complex128)
    if not c:
        if len(t) == 1:
            L.dense1(t[0], _ptr(m), _ptr(state), dim)
        elif len(t) == 2:
            L.dense2(t[0], t[1], _ptr(m), _ptr(state), dim)
        else:
            ta = np.asarray(t, dtype=np.uint32)
            L.dense_multi(_ptr(ta), len(t), _ptr(m), _ptr(state), dim)
        return
    ca = np.asarray(c, dtype=np.uint32)
    va = np.asarray(cv, dtype=np.uint32)
    ta = np.asarray(t, dtype=np.uint32)
    L.controlled(_ptr(ca), _ptr(va), len(c), _ptr(ta), len(t), _ptr(m), _ptr(state), dim)


def apply_gates(state: np.ndarray, gates: Sequence) -> np.ndarray:
    for g in gates:
        apply_gate(state, g)
    return state


def run_circuit(n: int, gates: Sequence, init: np.ndarray | None = None) -> np.ndarray:
    s = zero_state(n) if init is None else np.array(init, dtype=np.complex128, copy=True)
    return apply_gates(s, gates)


def norm_squared(state: np.ndarray) -> float:
    return float(lib().norm_squared(_ptr(state), state.size))


def inner_product(bra: np.ndarray, ket: np.ndarray) -> complex:
    out = np.zeros(2)
    lib().inner_product(_ptr(bra), _ptr(ket), bra.size, _ptr(out))
    return complex(out[0], out[1])


def max_threads() -> int:
    return int(lib().max_threads())
