"""Packing of gate objects for the engine (qulacs._native.make_gate_array): any
object with the public accessors is taken at its word, inverses included."""
import ctypes as ct

import numpy as np
import pytest

from qulacs import _native, gate as G
from qulacs._gates import ParametricRotationGate, QuantumGateMatrix

MATRIX = np.array([[0.6, 0.8j], [0.8j, 0.6]])


class AccessorsOnly:
    """No base class of this package."""

    def get_name(self):
        return "Own"

    def get_target_index_list(self):
        return [3]

    def get_control_index_list(self):
        return [1]

    def get_control_value_list(self):
        return [0]

    def get_matrix(self):
        return MATRIX.copy()


class Relabelled(QuantumGateMatrix):
    def get_target_index_list(self):
        return [q + 2 for q in super().get_target_index_list()]

    def get_control_index_list(self):
        return [q + 1 for q in super().get_control_index_list()]

    def get_control_value_list(self):
        return [1 - v for v in super().get_control_value_list()]

    def get_matrix(self):
        return -super().get_matrix()


def relabelled():
    g = Relabelled([0], MATRIX)
    g.add_control_qubit(4, 1)
    return g


def own_accessor():
    g = G.RX(1, 0.3)
    g.get_target_index_list = lambda: [5]
    return g


def own_matrix():
    g = G.DenseMatrix([0, 2], np.eye(4))
    g.get_matrix = lambda: np.diag([1, 1j, -1, -1j])
    return g


class Phased(ParametricRotationGate):
    """exp(i theta) times the rotation: its inverse is not read off one matrix
    alone but asked for."""

    def get_matrix(self):
        return np.exp(1j * self._angle) * super().get_matrix()


class Shifted(ParametricRotationGate):
    """Setting the angle adds a quarter turn, so get_inverse() is no dagger."""

    def set_parameter_value(self, value):
        super().set_parameter_value(value + np.pi / 2)


class OwnInverse(QuantumGateMatrix):
    def get_inverse(self):
        return G.X(0)


CASES = [AccessorsOnly, relabelled, own_accessor, own_matrix, lambda: Phased("Y", 2, 0.7), lambda: Shifted("Z", 1, 0.4),
         lambda: OwnInverse([1], MATRIX), lambda: ParametricRotationGate("X", 0, 1.1), lambda: G.CNOT(2, 0),
         lambda: G.SWAP(1, 3)]


def check(rec, g):
    t, c, v = g.get_target_index_list(), g.get_control_index_list(), g.get_control_value_list()
    m = np.asarray(g.get_matrix(), dtype=np.complex128).reshape(-1)
    assert rec.name == g.get_name().encode() and rec.ntargets == len(t) and rec.ncontrols == len(c)
    assert list(rec.targets) == t + [0] * (2 - len(t))
    assert list(rec.controls) == c + [0] * (2 - len(c))
    assert list(rec.control_values) == v + [0] * (2 - len(v))
    assert np.array_equal(np.array(rec.matrix[:2 * m.size]).view(np.complex128), m)


@pytest.mark.parametrize("make", CASES)
def test_packed_gate_is_what_its_accessors_say(make):
    arr = _native.make_gate_array([G.H(0), make()])
    check(arr[0], G.H(0))
    check(arr[1], make())


@pytest.mark.parametrize("make", CASES[3:])
def test_packed_inverse_is_what_get_inverse_says(make):
    from qulacs.torch import _inverse_gate_array
    arr = _inverse_gate_array([make(), G.T(1)])
    check(arr[0], make().get_inverse())
    check(arr[1], G.T(1).get_inverse())


@pytest.mark.parametrize("index", [-1, 1 << 31, (1 << 32) - 1])
def test_index_of_no_qubit_is_the_engines_to_refuse(index):
    L = _native.load_library()
    g = G.DenseMatrix(index, np.eye(2))
    arr = _native.make_gate_array([G.H(0), g])
    assert arr[1].targets[0] == index % (1 << 32)
    ns = ct.c_size_t()
    assert L.qs_plan_stages(arr, 2, 6, 4, 1, ct.byref(ns), None, None, None, None) == _native.QS_ERR_ARG
    assert b"range" in L.qs_last_error(None)
