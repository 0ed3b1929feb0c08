"""Gate takes its angles and qubits as any sequence (host only)."""
import numpy as np
import pytest

from spinoza_gb300 import _native as nat
from spinoza_gb300.gates import Gate


@pytest.mark.parametrize("form", [list, tuple, np.array])
def test_any_sequence(form):
    g = Gate(nat.SWAP, qubits=form([3, 1]))
    assert g.qubits == (3, 1) and g.params == (0.0, 0.0, 0.0)
    assert all(type(q) is int for q in g.qubits)
    assert Gate(nat.SWAP, qubits=form([2])).qubits == (2, 0)
    assert Gate(nat.H, qubits=form([])).qubits == (0, 0)
    assert Gate(nat.P, form([0.25])).params == (0.25, 0.0, 0.0)
    assert Gate(nat.U, form([0.25, 0.5, 1.0])).params == (0.25, 0.5, 1.0)
    assert Gate(nat.H, form([])).params == (0.0, 0.0, 0.0)
