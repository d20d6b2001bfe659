"""A complex64 trajectory whose norm has drifted when a known qubit is measured again (here by 2 %, far more than
FP32 rounding does): the next outcome is drawn from the state's own weights, and the state is of norm one
after it, as when the known qubit's measurement divided by the norm."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from lucivant_sim_gb300 import _lib, gates
from lucivant_sim_gb300.trajectories import TrajectoryProgram

pytestmark = pytest.mark.gpu


def _gate(m, q):
    return SimpleNamespace(kind="gate", name="g", matrix=np.asarray(m, dtype=complex), qubits=[q])


def _measure(q, clbit):
    return SimpleNamespace(kind="measure", qubit=q, clbit=clbit)


class _Noise:
    """Amplitude damping after gates named "k"."""

    def gate_error(self, name, qubits):
        if name != "k":
            return None
        g = 0.5
        return SimpleNamespace(mixture=None, kraus=[np.array([[0, np.sqrt(g)], [0, 0]]), np.diag([1, np.sqrt(1 - g)])])

    def readout_error(self, qubit):
        return None


def _run(n, ops, uniforms, members=1, noise=None):
    circuit = SimpleNamespace(num_qubits=n, num_clbits=8, operations=ops)
    program = TrajectoryProgram(circuit, noise, _lib.C64, members)
    try:
        u = np.zeros((members, program.max_draws))
        u[:, : len(uniforms)] = uniforms
        if members == 1:
            rows, _, _ = program.run_serial(1, u[0])
        else:
            rows, _, _ = program.run_batched(u)
        return int(rows[0, 0]), np.sum(np.abs(program.reg.download()) ** 2, axis=1)
    finally:
        program.free()


@pytest.mark.parametrize("members", [1, 3])
@pytest.mark.parametrize("n", [2, 3, 9, 13])
@pytest.mark.parametrize("target", [0, 1])
def test_the_next_outcome_is_drawn_from_the_states_weights(n, target, members):
    other = 1 - target
    p1 = float(np.sin(0.6) ** 2)
    grow = _gate(np.eye(2) * np.sqrt(1.02), other)
    grow.matrix[1, 1] *= 1j  # a diagonal, which leaves `other` known
    ops = [_gate(gates.ry(1.2), target), _measure(other, 0), grow, _measure(other, 1), _measure(target, 2)]
    for uniform, want in ((p1 * 0.999, 1), (p1 * 1.01, 0)):
        # (a barrier keeps the measurements of the batch from being one group)
        bits, norms = _run(n, [*ops[:4], _gate(np.diag([1, 1j]), target), ops[4]], [0.5, 0.5, uniform], members)
        assert bits >> 2 == want
        assert np.all(np.abs(norms - 1) < 1e-6)


@pytest.mark.parametrize("n", [2, 9])
def test_kraus_branches_are_drawn_from_the_states_weights(n):
    grow = _gate(np.diag([1, 1j]) * np.sqrt(1.02), 1)
    damp = _gate(np.diag([1, 1j]), 0)
    damp.name = "k"
    ops = [_gate(gates.ry(1.2), 0), _measure(1, 0), grow, _measure(1, 1), damp]
    weight = 0.5 * float(np.sin(0.6) ** 2)  # of the decay
    for uniform, decays in ((weight * 0.999, True), (weight * 1.01, False)):
        bits, norms = _run(n, [*ops, _measure(0, 2)], [0.5, 0.5, uniform, 1e-9], noise=_Noise())
        # decayed: qubit 0 is 0; not: a uniform near 0 finds 1
        assert (bits >> 2 == 0) == decays
        assert np.all(np.abs(norms - 1) < 1e-6)
