"""Small states are made from the handles of destroyed ones: what the last owner
did (lazy gates left pending, tile geometry, grown scratch, other streams, work
vectors) does not reach the next."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import adjoint, core, gates, rng
from spinoza_gb300.circuit import QuantumCircuit, QuantumRegister
from spinoza_gb300.core import State
from spinoza_gb300.gates import Gate

pytestmark = pytest.mark.gpu


def _lazy(s):
    s.set_lazy(True)
    for q in range(s.n):
        gates.apply(Gate.RY(0.3 + q), s, q)  # the carried factor is left pending


def _tile(s):
    s.set_tile(6 if s.n >= 6 else 4, 32)
    QuantumCircuit.from_state(s, fast=True).execute_ops(adjoint.hardware_efficient_ansatz(s.n, 1)[0])


def _scratch(s):
    core.sample(s, rng.uniforms(1, 200_000))  # more scratch than a kept handle may have


def _few_shots(s):
    core.sample(s, rng.uniforms(1, 100))


def _other_stream(s):
    import torch

    s.set_stream(torch.cuda.Stream())
    for q in range(s.n):
        gates.apply(Gate.H, s, q)


def _arrays(s):
    s.device_arrays()
    gates.apply(Gate.X, s, 0)


def _copied(s):
    _copied.other = s.clone()


def _work_vectors(s):
    ops, params = adjoint.hardware_efficient_ansatz(s.n, 1)
    adjoint.adjoint_gradient(s, ops, params, core.ising_hamiltonian(np.ones(s.n - 1), np.ones(s.n)))


def _measured(s):
    qc = QuantumCircuit.from_state(s, seed=2)
    qc.h(0)
    qc.measure(0)
    qc.x(1)
    qc.execute()


@pytest.mark.parametrize("use", [_lazy, _tile, _scratch, _few_shots, _other_stream, _arrays, _copied, _work_vectors, _measured])
@pytest.mark.parametrize("n", [2, 10, 14])
def test_a_new_state_is_as_new(gpu, n, use):
    for _ in range(3):
        s = State.from_arrays(*rng.normal_state(n, 7))
        use(s)
        del s
        t = State(n)
        re, im = t.to_numpy()
        assert re[0] == 1.0 and not np.any(re[1:]) and not np.any(im)
        init = rng.normal_state(n, 8)
        t.upload(*init)
        ore, oim = init[0].copy(), init[1].copy()
        for q, g in enumerate((Gate.H, Gate.RX(0.4))):  # exact arithmetic, not lazy
            gates.apply(g, t, q)
            oracle.apply(oracle.gate(g.kind, g.params), ore, oim, q)
        got = t.to_numpy()
        assert np.array_equal(got[0], ore) and np.array_equal(got[1], oim)
        del t


def test_many_states_at_once_share_nothing(gpu):
    states = [State(6) for _ in range(12)]
    for k, s in enumerate(states):
        gates.apply(Gate.RY(0.1 * k), s, k % 6)
    del states[3:9]
    more = [State(6) for _ in range(8)]
    for k, s in enumerate(more):
        assert s.to_numpy()[0][0] == 1.0
        gates.apply(Gate.X, s, k % 6)
    for k, s in zip((0, 1, 2, 9, 10, 11), states):
        re, im = oracle.zero_state(6)
        oracle.apply(oracle.gate(Gate.RY(0.1 * k).kind, Gate.RY(0.1 * k).params), re, im, k % 6)
        assert np.array_equal(s.to_numpy()[0], re)
    qc = QuantumCircuit(QuantumRegister(6))
    qc.x(2)
    qc.execute()
    assert qc.get_statevector().to_numpy()[0][4] == 1.0
