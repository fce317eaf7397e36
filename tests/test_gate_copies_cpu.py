"""Shallow copies of parametrised gates: a subclass with slots or with its own way
of being copied keeps its state, as through ``copy.copy``; the package's own gates share their matrix."""
import numpy as np
import pytest
import torch

from qaravan_gb300 import gates
from qaravan_gb300.circuits import Circuit
from qaravan_gb300.gates import RY, ParamGate


class Slotted(RY):
    __slots__ = ("tag",)


class OwnCopy(RY):
    def __copy__(self):
        g = type(self).__new__(type(self))
        g.__dict__.update(self.__dict__)
        g.copies = getattr(self, "copies", 0) + 1
        return g


class OwnState(RY):
    def __getstate__(self):
        return dict(self.__dict__, seen=True)


@pytest.mark.parametrize("angle", [0.3, torch.tensor(0.3, dtype=torch.float64)])
def test_subclasses_keep_their_state(angle):
    a, b, c = Slotted([0], angle), OwnCopy([1], angle), OwnState([0], angle)
    a.tag = "kept"
    circ = Circuit([a, b, c], n=2).copy()
    x, y, z = circ.gate_list
    assert (type(x), x.tag, x.indices) == (Slotted, "kept", [0])
    assert (type(y), y.copies, y.indices) == (OwnCopy, 1, [1])
    assert (type(z), z.seen) == (OwnState, True)
    for g in (x, y, z):
        assert np.allclose(np.asarray(g.matrix), [[np.cos(0.3), -np.sin(0.3)], [np.sin(0.3), np.cos(0.3)]])


@pytest.mark.parametrize("cls", sorted(gates._PLAIN_GATES, key=lambda c: c.__name__))
def test_own_gates_are_their_dict(cls):
    assert issubclass(cls, ParamGate) and not any("__slots__" in c.__dict__ for c in cls.__mro__)
    assert not any(hasattr(cls, m) for m in ("__copy__", "__setstate__"))
    angles = (0.3, 0.2, 0.1) if cls is gates.U else (0.3,) * (3 if cls is gates.HeisenbergCoupling else 1)
    try:
        g = cls([0, 1] if cls.__name__ not in ("RX", "RY", "RZ", "U") else [0], *angles)
    except Exception as e:  # (an angle count of its own)
        pytest.skip(str(e))
    h = g.shallow_copy()
    assert type(h) is cls and h.matrix is g.matrix and h.indices == g.indices and h.indices is not g.indices
