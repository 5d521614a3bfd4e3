"""What Orkan.gate takes as qubits and angles, on functions that record their arguments (no device)."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from orkan_b200 import Orkan, StateT

P = C.POINTER(StateT)


@pytest.fixture
def ork():
    seen = []

    class Lib:
        pass

    def bind(name, *types):
        fn = C.CFUNCTYPE(None, P, *types)(lambda s, *a: seen.append((name,) + a))
        fn.argtypes = [P, *types]
        return fn

    o = object.__new__(Orkan)
    o.lib = Lib()
    o._gates = {"x": bind("x", C.c_ubyte), "rx": bind("rx", C.c_ubyte, C.c_double), "swap": bind("swap", C.c_ubyte, C.c_ubyte)}
    o.lib.swap_gate = o._gates["swap"]
    o.seen = seen
    return o


QUBITS = [[5, 2], (5, 2), np.array([5, 2]), np.array([5.0, 2.0]), [np.uint8(5), np.float32(2)], (5.0, "2"), range(5, 1, -3)]


@pytest.mark.parametrize("qubits", QUBITS, ids=str)
@pytest.mark.parametrize("form", [lambda q: q, iter, lambda q: (x for x in q)], ids=["as is", "iterator", "generator"])
@pytest.mark.parametrize("name", ["swap", "swap_gate"])
def test_qubits(ork, qubits, form, name):
    ork.gate(StateT(0, None, 8), name, form(qubits))
    assert ork.seen == [("swap", 5, 2)]


@pytest.mark.parametrize("theta", [0.25, np.float32(0.25), np.float64(0.25), Fraction(1, 4), "0.25", np.array(0.25)], ids=repr)
def test_angles(ork, theta):
    s = StateT(0, None, 8)
    ork.gate(s, "rx", (x for x in (3.0,)), theta)
    ork.gate(s, "rx", [3], theta)
    assert ork.seen == [("rx", 3, 0.25)] * 2


def test_wrong_counts_and_names_are_refused(ork):
    s = StateT(0, None, 8)
    with pytest.raises(TypeError):
        ork.gate(s, "rx", [3])
    with pytest.raises(TypeError):
        ork.gate(s, "x", [])
    with pytest.raises(AttributeError):
        ork.gate(s, "nothing", [0])
    with pytest.raises((TypeError, ValueError)):
        ork.gate(s, "x", ["a"])
    assert ork.seen == []
